// fp32 filter gradient with the operands converted on the way in: U[(c,r,s), k] = sum over (p,q,n) of
// I[c, p*str-pad+r, q*str-pad+s, n] * E[k, p, q, n], 3xTF32 as in b2_direct.cuh.
//
// Operands as in the flex16 filter gradient (b2_conv.cu): a k-block is a tile of gh x gw output pixels
// times 32 images; A has a row for every (channel, place in the window under the tile), B one for every
// (filter, pixel), and the epilogue adds the pixels' shares of a tap.  Eight producer warps load the
// rows (32 images: 128 contiguous bytes), split them into two tf32 planes and store them into a ring;
// a ninth issues the products.  A slice of at most 16 k-blocks goes to each CTA (the tensor core's fp32
// sum truncates: a longer chain would lose what 3xTF32 gains); its sums go to partial[slice], which
// update_f32_finish_kernel adds in slice order.  A slice's sums are a copy of the filters, and slices are
// as many as the pixels and images ask for, so they go in rounds of what kScratchMost holds: 512 -> 512
// channels, 3x3, 56x56 pixels of 256 images have 784 slices, 7.4 GB at once, in 28 rounds (of 11648 CTAs
// each, 79 to an SM, so that the ends of the rounds cost little).  512 -> 512 channels, 3x3, 28x28 pixels
// of 128 images: 10.59 ms with 1.8 GB of slices, 10.39 in seven rounds.
//
// What bounds it: the producers' issue slots, so a window is loaded once for up to four pixels.  The
// unrolled planes and their product took 1.4 ms of a batch-128 training step of ResNet-14.
#include "b2_direct.cuh"

namespace {

struct UpdF32Params {
    b2_update_f32 g;
    const float *I, *E;
    float* partial;                    // [slice][C*R*S][K]
    int gh, gw, wh, ww, cu, ntn, kt, tw, nblk, nkb, per, slice0;
    int vec;                           // rows start on 16-byte boundaries
    int* status;
};

template <int BN>
__global__ void __launch_bounds__(kDirThreads, (BN == 128 ? 1 : 2))
conv_update_f32_kernel(const __grid_constant__ UpdF32Params p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int NST = dir_stages(BN), STAGE = dir_stage_bytes(BN);
    constexpr int kCols = dir_tmem_cols(MODE_F32X3, BN);
    typedef OperandTile<MODE_F32X3, 128> ATile;
    typedef OperandTile<MODE_F32X3, BN> BTile;
    unsigned long long* full_bar = (unsigned long long*)(smem + NST * STAGE);
    unsigned long long* empty_bar = full_bar + NST;
    unsigned long long* tmem_full = empty_bar + NST;
    unsigned* tmem_holder = (unsigned*)(tmem_full + 1);
    int* fail_flag = (int*)(tmem_holder + 1);

    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const b2_update_f32& g = p.g;
    const int chunk = blockIdx.y / p.ntn, ktile = blockIdx.y - chunk * p.ntn;
    const int kb0 = (p.slice0 + blockIdx.x) * p.per, nkb = min(p.per, p.nkb - kb0);
    const int win = p.wh * p.ww, npix = p.gh * p.gw;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NST; ++s) { mbar_init(&full_bar[s], 8); mbar_init(&empty_bar[s], 1); }
        mbar_init(tmem_full, 1);
        *fail_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        tmem_alloc(tmem_holder, kCols);
        // (not before this CTA holds its tensor memory, or it and the next kernel's could each wait for
        // what the other has)
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = (unsigned)warp_uniform((int)*tmem_holder);

    if (warp < 8) {
        // ---- producers: place of each of this lane's rows, in values from the tile's corner
        ATile ta[2];
        BTile tb[2];
        int a_dh[ATile::kKUnits], a_dw[ATile::kKUnits], b_dh[BTile::kKUnits], b_dw[BTile::kKUnits];
        long long a_base[ATile::kKUnits], b_base[BTile::kKUnits];
#pragma unroll
        for (int i = 0; i < ATile::kKUnits; ++i) {
            const int lr = (warp + 8 * i) * 4 + (lane >> 3), c = lr / win, at = lr - c * win;
            const int cg = chunk * p.cu + c;
            a_dh[i] = at / p.ww; a_dw[i] = at - a_dh[i] * p.ww;
            a_base[i] = (((long long)cg * g.H + a_dh[i]) * g.W + a_dw[i]) * g.N + (lane & 7) * 4;
            if (c >= p.cu || cg >= g.C) a_dh[i] = 1 << 28;                // no such row
        }
#pragma unroll
        for (int i = 0; i < BTile::kKUnits; ++i) {
            const int lr = (warp + 8 * i) * 4 + (lane >> 3), k = lr / npix, pix = lr - k * npix;
            const int kg = ktile * p.kt + k;
            b_dh[i] = pix / p.gw; b_dw[i] = pix - b_dh[i] * p.gw;
            b_base[i] = (((long long)kg * g.P + b_dh[i]) * g.Q + b_dw[i]) * g.N + (lane & 7) * 4;
            if (k >= p.kt || kg >= g.K) b_dh[i] = 1 << 28;
        }
        int nb = kb0 % p.nblk, q = kb0 / p.nblk % p.tw, pp = kb0 / p.nblk / p.tw;      // the next load's
        auto load = [&](ATile& A, BTile& B) {
            const int h0 = pp * p.gh * g.str_h - g.pad_h, w0 = q * p.gw * g.str_w - g.pad_w, n0 = nb * 32;
            const long long a_off = ((long long)h0 * g.W + w0) * g.N + n0;
            const long long b_off = ((long long)pp * p.gh * g.Q + q * p.gw) * g.N + n0;
            long long a_at[ATile::kKUnits], b_at[BTile::kKUnits];
#pragma unroll
            for (int i = 0; i < ATile::kKUnits; ++i)
                a_at[i] = (unsigned)(h0 + a_dh[i]) < (unsigned)g.H && (unsigned)(w0 + a_dw[i]) < (unsigned)g.W
                              ? (a_base[i] + a_off) * 4 : -1;
#pragma unroll
            for (int i = 0; i < BTile::kKUnits; ++i)
                b_at[i] = pp * p.gh + b_dh[i] < g.P && q * p.gw + b_dw[i] < g.Q ? (b_base[i] + b_off) * 4 : -1;
            A.load_k(p.I, a_at, 0, g.N - n0, p.vec, lane);
            B.load_k(p.E, b_at, 0, g.N - n0, p.vec, lane);
            if (++nb == p.nblk) {
                nb = 0;
                if (++q == p.tw) { q = 0; ++pp; }
            }
        };
        load(ta[0], tb[0]);
        int s = 0;
        unsigned parity = 1;
        bool ok = true;
        auto put = [&](int kb, ATile& A, BTile& B, ATile& An, BTile& Bn) {
            if (kb + 1 < nkb) load(An, Bn);                              // in flight while this one is stored
            if (ok && !mbar_wait(&empty_bar[s], parity)) { atomicExch(fail_flag, 1); ok = false; }
            unsigned char* st = smem + s * STAGE;
            A.store_k(st, st + 128 * 128, warp, lane);
            B.store_k(st + 2 * 128 * 128, st + 2 * 128 * 128 + BN * 128, warp, lane);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_bar[s]);
            if (++s == NST) { s = 0; parity ^= 1u; }
        };
        for (int kb = 0; kb < nkb; kb += 2) {
            put(kb, ta[0], tb[0], ta[1], tb[1]);
            if (kb + 1 < nkb) put(kb + 1, ta[1], tb[1], ta[0], tb[0]);
        }
    } else if (elect_one()) {
        // ---- MMA issue: A_hi x [B_hi | B_lo] -> [hh | x], A_lo x B_hi -> x
        const unsigned id_t1 = make_idesc(1, 2, 2, BN), id_t2 = make_idesc(1, 2, 2, 2 * BN);
        int s = 0;
        unsigned parity = 0;
        for (int kb = 0; kb < nkb; ++kb) {
            if (!mbar_wait(&full_bar[s], parity)) { atomicExch(fail_flag, 1); break; }
            tc_fence_after();
            unsigned char* st = smem + s * STAGE;
            const unsigned long long dA0 = make_smem_desc(st), dA1 = make_smem_desc(st + 128 * 128);
            const unsigned long long dB0 = make_smem_desc(st + 2 * 128 * 128);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const unsigned long long adv = (unsigned long long)(2 * k);
                tc_mma<MODE_F32X3>(tmem_base, dA0 + adv, dB0 + adv, id_t2, (kb > 0 || k > 0) ? 1u : 0u);
                tc_mma<MODE_F32X3>(tmem_base + BN, dA1 + adv, dB0 + adv, id_t1, 1u);
            }
            tc_commit(&empty_bar[s]);
            if (++s == NST) { s = 0; parity ^= 1u; }
        }
        tc_commit(tmem_full);
    }
    __syncwarp();

    // ---- epilogue (warps 0-7): tensor memory -> shared memory [row][column], then per tap
    float* red = (float*)smem;
    constexpr int pitch = BN + 1;
    if (warp < 8) {
        const int row = (warp & 3) * 32 + lane;
        if (!mbar_wait(tmem_full, 0)) atomicExch(fail_flag, 1);
        tc_fence_after();
        const unsigned lane_addr = tmem_base + ((unsigned)((warp & 3) * 32) << 16);
        for (int c0 = (warp >> 2) * 8; c0 < BN; c0 += 16) {
            unsigned hh[8], xx[8];
            tmem_ld8(lane_addr + c0, hh);
            tmem_ld8(lane_addr + BN + c0, xx);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 8; ++j)
                red[row * pitch + c0 + j] = __uint_as_float(hh[j]) + __uint_as_float(xx[j]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kCols);
    }
    const int rs = g.R * g.S, rows = min(p.cu, g.C - chunk * p.cu) * rs;
    float* out = p.partial + ((long long)blockIdx.x * g.C + chunk * p.cu) * rs * g.K + ktile * p.kt;
    if (*fail_flag == 0)
        for (int i = threadIdx.x; i < rows * p.kt; i += kDirThreads) {
            const int t = i / p.kt, k = i - t * p.kt, c = t / rs, tap = t - c * rs, r = tap / g.S, s = tap - r * g.S;
            if (ktile * p.kt + k >= g.K) continue;
            const float* at = red + ((c * p.wh + r) * p.ww + s) * pitch + k * npix;
            float v = 0.0f;
            for (int a = 0; a < p.gh; ++a)
                for (int b = 0; b < p.gw; ++b) v += at[(a * g.str_h * p.ww + b * g.str_w) * pitch + a * p.gw + b];
            out[(long long)t * g.K + k] = v;
        }
    if (threadIdx.x == 0 && *fail_flag && p.status) atomicExch(p.status, 1);
}

// Sum of the slices, in a fixed order: a block has 32 outputs, warp w adds the slices w, w+8, ... (four
// loads in flight), then the eight sums are added in warp order.  add: to what earlier rounds left.
__global__ void __launch_bounds__(256)
update_f32_finish_kernel(const float* __restrict__ partial, float* __restrict__ U, int n, int slices, int add) {
    after_earlier_kernels();
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    float v = 0.0f;
    if (i < n) {
        int z = w;
        for (; z + 24 < slices; z += 32) {
            float x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = __ldcg(partial + (long long)(z + 8 * j) * n + i);
#pragma unroll
            for (int j = 0; j < 4; ++j) v += x[j];
        }
        for (; z < slices; z += 8) v += __ldcg(partial + (long long)z * n + i);
    }
    part[w][lane] = v;
    __syncthreads();
    if (w == 0 && i < n) {
#pragma unroll
        for (int j = 1; j < 8; ++j) v += part[j][lane];
        U[i] = add ? U[i] + v : v;
    }
}

const size_t kScratchMost = 256u << 20;

struct UpdF32Shape { bool ok; int gh, gw, wh, ww, cu, cchunks, ntn, kt, bn, tw, nblk, nkb, per, nsplit, round; long long cost; };

UpdF32Shape update_f32_shape_for(const b2_update_f32& g, int gh, int gw) {
    UpdF32Shape u = {};
    u.gh = gh; u.gw = gw; u.wh = (gh - 1) * g.str_h + g.R; u.ww = (gw - 1) * g.str_w + g.S;
    const int win = u.wh * u.ww, npix = gh * gw;
    const long long nkb = (long long)((g.P + gh - 1) / gh) * ((g.Q + gw - 1) / gw) * ((g.N + 31) / 32);
    if (win > 128 || nkb >= (1LL << 24)) return u;
    u.tw = (g.Q + gw - 1) / gw; u.nblk = (g.N + 31) / 32; u.nkb = (int)nkb;
    const int cu_max = 128 / win, kt_max = 128 / npix;
    u.cchunks = (g.C + cu_max - 1) / cu_max;
    u.cu = (g.C + u.cchunks - 1) / u.cchunks;
    u.ntn = (g.K + kt_max - 1) / kt_max;
    u.kt = (g.K + u.ntn - 1) / u.ntn;
    u.bn = 16;
    while (u.bn < u.kt * npix) u.bn *= 2;
    const long long cols = (long long)u.cchunks * u.ntn;
    if (cols > 65535) return u;
    // a slice for every CTA that the SMs hold at once, or a multiple where one would exceed 16 k-blocks
    const int slots = u.bn == 128 ? 148 : 296;
    long long slices = cols < slots ? slots / cols : 1;
    const long long per = (nkb + slices - 1) / slices;
    slices *= (per + 15) / 16;
    u.per = (int)((nkb + slices - 1) / slices);
    u.nsplit = (int)((nkb + u.per - 1) / u.per);
    const long long filters = (long long)g.C * g.R * g.S * g.K;
    if (u.nsplit * filters >= (1LL << 31)) return u;
    const long long fit = (long long)(kScratchMost / 4) / filters;
    u.round = fit < 1 ? 1 : fit < u.nsplit ? (int)fit : u.nsplit;
    // cycles: the producers' 7 a row of a k-block (two CTAs of an SM share them), the sums' way out
    const long long waves = (cols * u.nsplit + slots - 1) / slots;
    u.cost = waves * ((long long)u.per * (300 + 7 * (128 + u.bn) * (slots / 148)) + 6000 + 60 * u.bn) +
             u.nsplit * 40LL;
    u.ok = true;
    return u;
}

UpdF32Shape update_f32_shape(const b2_update_f32& g) {
    UpdF32Shape best = {};
    for (int gh = 1; gh <= 2; ++gh)
        for (int gw = 1; gw <= 2; ++gw) {
            const UpdF32Shape u = update_f32_shape_for(g, gh, gw);
            if (u.ok && (!best.ok || u.cost < best.cost)) best = u;
        }
    return best;
}

template <int BN>
int launch_update_f32(const UpdF32Params& p, const UpdF32Shape& u, int slices, cudaStream_t st) {
    static_assert(dir_ring_bytes(BN) >= 128 * (BN + 1) * 4, "the sums fit the ring");
    const int smem = 1024 + dir_ring_bytes(BN) + 128;
    static bool attr_set = false;
    if (!attr_set) {
        B2_CUDA(cudaFuncSetAttribute(conv_update_f32_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attr_set = true;
    }
    B2_CUDA(b2::launch_after(conv_update_f32_kernel<BN>, dim3(slices, u.cchunks * u.ntn), kDirThreads, smem, st, p));
    return B2_OK;
}

}  // namespace

size_t b2_update_f32_scratch(const b2_update_f32& g) {
    const UpdF32Shape u = update_f32_shape(g);
    return u.ok ? (((size_t)u.round * g.C * g.R * g.S * g.K * 4) + 1023) / 1024 * 1024 : 0;
}

int b2_update_f32_launches(const b2_update_f32& g) {
    const UpdF32Shape u = update_f32_shape(g);
    return !u.ok ? 0 : u.nsplit == 1 ? 1 : 2 * ((u.nsplit + u.round - 1) / u.round);
}

int b2_update_f32_launch(const b2_update_f32& g, const float* I, const float* E, float* U, void* scratch,
                         int* status, cudaStream_t st) {
    const UpdF32Shape u = update_f32_shape(g);
    B2_REQUIRE(u.ok, "problem outside the kernel's range");
    UpdF32Params p;
    p.g = g; p.I = I; p.E = E; p.partial = u.nsplit > 1 ? (float*)scratch : U;
    p.gh = u.gh; p.gw = u.gw; p.wh = u.wh; p.ww = u.ww; p.cu = u.cu; p.ntn = u.ntn; p.kt = u.kt;
    p.tw = u.tw; p.nblk = u.nblk; p.nkb = u.nkb; p.per = u.per; p.status = status;
    p.vec = g.N % 4 == 0 && (((uintptr_t)I | (uintptr_t)E) & 15) == 0;
    const int n = g.C * g.R * g.S * g.K;
    for (p.slice0 = 0; p.slice0 < u.nsplit; p.slice0 += u.round) {
        const int slices = u.nsplit - p.slice0 < u.round ? u.nsplit - p.slice0 : u.round;
        int rc;
        switch (u.bn) {
            case 16: rc = launch_update_f32<16>(p, u, slices, st); break;
            case 32: rc = launch_update_f32<32>(p, u, slices, st); break;
            case 64: rc = launch_update_f32<64>(p, u, slices, st); break;
            default: rc = launch_update_f32<128>(p, u, slices, st); break;
        }
        if (rc || u.nsplit == 1) return rc;
        B2_CUDA(b2::launch_after(update_f32_finish_kernel, dim3((n + 31) / 32), 256, 0, st, (const float*)scratch, U, n,
                                 slices, p.slice0 > 0 ? 1 : 0));
    }
    return B2_OK;
}
