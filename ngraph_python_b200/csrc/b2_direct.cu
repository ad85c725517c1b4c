// Dispatch of the kernel with operands converted on the way in; the fp32 half of it.
#include <cmath>
#include "b2_direct.cuh"

__attribute__((visibility("hidden"))) int b2_direct_launch_flex(const b2_direct_args& a, cudaStream_t st);

static bool within_range(const b2_direct_args& a) {
    if (a.a_kind == B2_OPERAND_GATHER) {
        const b2_gather& g = a.g;
        const long long elems = (long long)g.channels * g.H * g.W * g.N;
        if (g.R * g.S > 31 || a.K > kDirMaxK || elems >= (1LL << 31)) return false;
    }
    return (long long)(a.M + 127) / 128 <= 65535;                  // grid.y
}

long long b2_direct_cost(const b2_direct_args& a) {
    if (!within_range(a)) return -1;
    if (b2_gather_streams(a)) return b2_gather_plan(a).cost;
    return a.flex ? direct_shape<MODE_FLEX16>(a).cost : direct_shape<MODE_F32X3>(a).cost;
}

long long b2_direct_longest(const b2_direct_args& a, int* longest) {
    if (!within_range(a)) return -1;
    const DirectShape s = direct_shape<MODE_F32X3>(a, true);
    *longest = s.kb_per_split;
    return s.cost;
}

int b2_direct_in_one_sum(const b2_direct_args& a) {
    if (b2_gather_streams(a)) return b2_gather_plan(a).in_one_sum;
    const DirectShape s = direct_shape<MODE_F32X3>(a);
    const int pairs = dir_pairs(s.bn, s.groups);
    return (s.kb_per_split + pairs - 1) / pairs;
}

double b2_direct_loss(const b2_direct_args& a) {
    const b2_gather& g = a.g;
    int per, splits, sums;
    if (b2_gather_streams(a)) {
        const b2_gather_info s = b2_gather_plan(a);
        per = s.kb_per_split; splits = s.splits; sums = s.sums;
    } else {
        const DirectShape s = direct_shape<MODE_F32X3>(a);
        per = s.kb_per_split; splits = s.splits; sums = dir_pairs(s.bn, s.groups);
    }
    const int taps = g.R * g.S, pixels = filter_tiles(a) ? g.gh * g.gw : 1;
    double lost = 0;
    for (int pixel = 0; pixel < pixels; ++pixel) {
        unsigned char seen[32];                   // (taps <= 31)
        for (int t = 0; t < taps; ++t) {
            const int r = g.f0_h + g.f1_h * (t / g.S) + g.f2_h * (pixel / g.gw), s = g.f0_w + g.f1_w * (t % g.S) + g.f2_w * (pixel % g.gw);
            seen[t] = !filter_tiles(a) || (r >= 0 && r < g.fr && s >= 0 && s < g.fs);
        }
        int tap = 0, channel = 0;                 // of the next column
        for (int z = 0; z < splits; ++z) {
            double sum[4] = {}, steps[4] = {};    // a sum's squared size; what its steps have cut off
            for (int kb = z * per; kb < (z + 1) * per && kb * 32 < a.K; ++kb)
                for (int step = 0; step < 4; ++step) {
                    int n = 0;
                    for (int k = kb * 32 + step * 8, end = k + 8; k < end && k < a.K; ++k) {
                        n += seen[tap];
                        if (g.channel_last) { if (++channel == g.channels) { channel = 0; ++tap; } }
                        else if (++tap == taps) tap = 0;
                    }
                    if (!n) continue;
                    const int i = (kb - z * per) % sums;
                    sum[i] += n;
                    steps[i] += sqrt(sum[i]);
                }
            for (int i = 0; i < sums; ++i) lost += steps[i] * steps[i];
        }
    }
    return lost / pixels;
}

void b2_direct_plan(const b2_direct_args& a, b2_gemm_plan_info* plan) {
    if (b2_gather_streams(a)) {
        const b2_gather_info s = b2_gather_plan(a);
        *plan = {B2_GEMM_DIRECT, s.bn, s.splits, s.waves};
        return;
    }
    const DirectShape s = a.flex ? direct_shape<MODE_FLEX16>(a) : direct_shape<MODE_F32X3>(a);
    *plan = {B2_GEMM_DIRECT, s.bn, s.splits, s.waves};
}

int b2_direct_launch(const b2_direct_args& a, cudaStream_t st) {
    B2_REQUIRE(b2_direct_cost(a) >= 0, "problem outside the kernel's range");
    if (b2_gather_streams(a)) return b2_gather_launch(a, st);
    return a.flex ? b2_direct_launch_flex(a, st) : direct_launch_mode<MODE_F32X3>(a, st);
}

// ---- filters as the stages hold them ------------------------------------------------------------
// The rows of the filters that the pixels of a tile see are the same in every tile, and making them costs
// a producer more than the rows it gathers (a lane's rows lie apart, each with its own tap): here each is
// made once, in the order n tile, k-block, plane, row, 128-byte swizzled, and the kernel copies a
// k-block's 2 * bn * 128 bytes as they are.  Bound by launch latency (a network's filters are some MB).
namespace {

struct StageLayout {
    const float* F;
    unsigned char* out;
    long long b_rs, b_ks;
    b2_gather g;
    int N, K, bn, num_kb, ntn, tiled, turned;       // turned: see b2_gather_info
};
struct StageJobs {
    int n, first[kStageJobs + 1];                 // job j owns blocks first[j] .. first[j+1]-1
    StageLayout layout[kStageJobs];
};
static_assert(sizeof(StageJobs) <= 4096, "kernel argument");

__global__ void __launch_bounds__(256)
stage_filters_kernel(const __grid_constant__ StageJobs jobs) {
    after_earlier_kernels();
    int j = 0;
    while (j + 1 < jobs.n && (int)blockIdx.x >= jobs.first[j + 1]) ++j;
    const StageLayout& f = jobs.layout[j];
    const b2_gather& g = f.g;
    const int RS = g.R * g.S, total = f.ntn * f.num_kb * 8 * f.bn;
    const int stride = (jobs.first[j + 1] - jobs.first[j]) * (int)blockDim.x;
    for (int i = ((int)blockIdx.x - jobs.first[j]) * (int)blockDim.x + threadIdx.x; i < total; i += stride) {
        const int lr = i % f.bn, chunk = i / f.bn % 8, block = i / f.bn / 8, kb = block % f.num_kb;
        const int row = block / f.num_kb * f.bn + lr;
        const int pix = f.tiled ? row / g.kt : 0, gy = f.tiled ? pix / g.gw : 0, gx = f.tiled ? pix - gy * g.gw : 0;
        float4 h, l;
        float *hp = (float*)&h, *lp = (float*)&l;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k = kb * 32 + chunk * 4 + q;
            float v = 0.0f;
            if (row < f.N && k < f.K) {
                if (f.tiled) {
                    const int c = g.channel_last ? k % g.channels : k / RS, rs = g.channel_last ? k / g.channels : k % RS;
                    const int th = rs / g.S, tw = rs - th * g.S;
                    const int r = g.f0_h + g.f1_h * th + g.f2_h * gy, s = g.f0_w + g.f1_w * tw + g.f2_w * gx;
                    if (r >= 0 && r < g.fr && s >= 0 && s < g.fs)
                        v = __ldg(f.F + c * f.b_ks + (row - pix * g.kt) * f.b_rs +
                                  (long long)(r * g.fs + s) * (g.channel_last ? g.channels : g.kt));
                } else {
                    v = __ldg(f.F + row * f.b_rs + k * f.b_ks);
                }
            }
            dir_split_tf32(v, hp[q], lp[q]);
        }
        unsigned char* out = f.out + (long long)block * (2 * f.bn * 128) + swz(lr, chunk);
        const bool turn = f.turned && (kb / f.turned & 1);
        *(float4*)out = turn ? l : h;
        *(float4*)(out + f.bn * 128) = turn ? h : l;
    }
}

}  // namespace

static int staged_tile(const b2_direct_args& a) {
    return b2_gather_streams(a) ? b2_gather_plan(a).bn : direct_shape<MODE_F32X3>(a).bn;
}

size_t b2_direct_staged_bytes(const b2_direct_args& a) {
    const int bn = staged_tile(a);
    return (size_t)((a.N + bn - 1) / bn) * ((a.K + 31) / 32) * (2 * bn * 128);
}

int b2_direct_stage_filters(const b2_stage_job* list, int n, int* launches, cudaStream_t st) {
    *launches = 0;
    for (int at = 0; at < n; at += kStageJobs) {
        StageJobs jobs = {};
        jobs.n = n - at < kStageJobs ? n - at : kStageJobs;
        for (int j = 0; j < jobs.n; ++j) {
            const b2_direct_args& a = list[at + j].a;
            const int bn = staged_tile(a), ntn = (a.N + bn - 1) / bn, num_kb = (a.K + 31) / 32;
            jobs.layout[j] = {list[at + j].filters, (unsigned char*)list[at + j].staged, a.b_rs, a.b_ks, a.g,
                              a.N, a.K, bn, num_kb, ntn, filter_tiles(a), b2_gather_streams(a) ? b2_gather_plan(a).turned : 0};
            const long long blocks = ((long long)ntn * num_kb * 8 * bn + 255) / 256;
            jobs.first[j + 1] = jobs.first[j] + (int)(blocks < 148 * 4 ? blocks : 148 * 4);
        }
        B2_CUDA(b2::launch_after(stage_filters_kernel, dim3(jobs.first[jobs.n]), 256, 0, st, jobs));
        B2_CUDA(cudaGetLastError());
        ++*launches;
    }
    return B2_OK;
}
