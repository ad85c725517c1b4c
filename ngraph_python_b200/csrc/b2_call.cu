// What a call of a compiled computation does around its kernels: taking the arguments in, handing
// the results out, and the exponent bookkeeping of every tensor it writes.
//
// Replaces the per-tensor host work of the reference's flex transformer -- one conversion and one
// upload per argument (ngraph/transformers/flexgputransform.py:178-208), one statistics read per
// kernel and manage_before / manage_after_computation per tensor (flexgputransform.py:347-371) --
// by one kernel at each end of a recorded step list and one pass over plain arrays on the host.
//
// k_call_inputs takes the arguments in.  The values are read from wherever they lie (the caller's own
// device tensor, the caller's pinned array, or the pinned block into which pageable memory was
// copied) and stored once, quantised where the tensor is flex16.  Bound by what it reads: PCIe for host
// arguments, HBM for device tensors.  A flex16 argument of 8192 x 16384 values: copy to a staging
// tensor 173 us + conversion 167 us before, one pass of 6 bytes a value now.
//
// b2_call_take launches it in front of a recorded step list: addresses and scales are launch parameters,
// only what is to be copied has blocks, and it runs while the launch of the graph is on its way (8 to
// 10 us from the call to the first node); pageable memory goes through the pinned block in pieces, each
// read by the device while the host copies the next.  As the graph's first node (b2_call_inputs) every block
// reads its addresses from pinned memory first, and the host has one launch less: the better way for few
// values (16 x 64 fp32 18.7 us a call, 21.2 in front).  A call, first node -> in front, one B200 under a host
// that launches slowly / quickly: 128 x 1000 fp32 values from the device 35 -> 24 / 26 -> 23 us, 400 KB pageable
// and 22 launches 149 -> 141, 3 MB pinned and a run of layers 249 -> 241 / 239 -> 242; 8192 x 16384 read in
// place by their kernel, flex16 / fp32 373 -> 355 / 538 -> 515.
#include <cmath>
#include <cstddef>
#include <cstring>
#if defined(__x86_64__)
#include <immintrin.h>
#endif

#include "b2_common.h"
#include "b2_ew_device.cuh"

namespace {

const int kThreads = 256;
// Values a thread takes from a chunk: 16, or 4 where that leaves too few blocks to keep PCIe busy
// (100 K values from the host: 22 us with 25 blocks of 4096 values)
const int kPerLong = 16, kPerShort = 4;

struct Inputs {
    int n;
    b2_call_input in[B2_CALL_MAX_INPUTS];
    long long first_chunk[B2_CALL_MAX_INPUTS + 1];
    // as of b2_call_take (else they stand in the block):
    const void* src[B2_CALL_MAX_INPUTS];      // nothing to copy where null
    float inv[B2_CALL_MAX_INPUTS];
    int n_words;                              // device words for addresses: where[i] <- address[i]
    const void** where[B2_CALL_MAX_INPUTS];
    const void* address[B2_CALL_MAX_INPUTS];
    const b2_flex_scale* rows;                // rows of the scale table
    int n_rows;
};

__device__ __forceinline__ short quant1(float x, float inv, int& stat) {
    const float v = fminf(fmaxf(x * inv, -32768.0f), 32767.0f);   // power-of-two scaling: exact
    const int m = (int)v;                                         // truncation toward zero
    stat = b2_absmax(stat, m);
    return (short)m;
}

template <int kPerThread>
__global__ void __launch_bounds__(kThreads)
k_call_inputs(const Inputs a, const b2_call_block* __restrict__ blk, b2_flex_scale* __restrict__ table,
              int* __restrict__ stats) {
    constexpr int kChunk = kThreads * kPerThread;
    after_earlier_kernels();
    __shared__ int ismem[32];
    __shared__ const float* src_s[B2_CALL_MAX_INPUTS];
    __shared__ float inv_s[B2_CALL_MAX_INPUTS];
    if (!blk) {
        if (threadIdx.x < a.n) {
            src_s[threadIdx.x] = (const float*)a.src[threadIdx.x];
            inv_s[threadIdx.x] = a.inv[threadIdx.x];
        }
        // (the last block has the fewest values to copy)
        if (blockIdx.x == gridDim.x - 1) {
            if (threadIdx.x < a.n_words) *a.where[threadIdx.x] = a.address[threadIdx.x];
            for (int i = threadIdx.x; i < a.n_rows; i += kThreads) table[i] = a.rows[i];
        }
    } else if (threadIdx.x < a.n) {
        // one 16-byte read over PCIe to a block and argument
        const uint4 e = *reinterpret_cast<const uint4*>(&blk->arg[threadIdx.x]);
        const float* src = (const float*)((unsigned long long)e.y << 32 | e.x);
        const bool in_place = src && e.w && a.in[threadIdx.x].where;
        src_s[threadIdx.x] = in_place ? nullptr : src;
        inv_s[threadIdx.x] = __uint_as_float(e.z);
        if (blockIdx.x == 0 && a.in[threadIdx.x].where)
            *a.in[threadIdx.x].where = in_place ? (const void*)src : a.in[threadIdx.x].dst;
    }
    // the scale table, when a row of it has changed
    if (blk && blockIdx.x == gridDim.x - 1 && table && blk->table_rows > 0) {
        const b2_flex_scale* h = blk->table;
        for (int i = threadIdx.x; i < blk->table_rows; i += kThreads) table[i] = h[i];
    }
    __syncthreads();
    int stat = 0, cur = 0;
    for (long long c = blockIdx.x; c < a.first_chunk[a.n]; c += gridDim.x) {
        int k = cur;
        while (c >= a.first_chunk[k + 1]) ++k;
        if (k != cur) {
            if (a.in[cur].flex_slot >= 0) b2_block_stat(stat, stats + a.in[cur].flex_slot, ismem);
            stat = 0;
            cur = k;
        }
        const float* src = src_s[k];
        if (!src) continue;                       // not an argument of this call: keep what is there
        const long long base = (c - a.first_chunk[k]) * kChunk;
        const long long left = a.in[k].n - base;
        const bool flex = a.in[k].flex_slot >= 0;
        const float inv = inv_s[k];
        if (left >= kChunk && (((uintptr_t)src | (uintptr_t)a.in[k].dst) & 15) == 0) {
            float4 v[kPerThread / 4];
            const float4* s4 = reinterpret_cast<const float4*>(src + base);
#pragma unroll
            for (int j = 0; j < kPerThread / 4; ++j) v[j] = __ldcs(s4 + j * kThreads + threadIdx.x);
            if (flex) {
                uint2* d = reinterpret_cast<uint2*>((short*)a.in[k].dst + base);
#pragma unroll
                for (int j = 0; j < kPerThread / 4; ++j) {
                    const unsigned short q0 = quant1(v[j].x, inv, stat), q1 = quant1(v[j].y, inv, stat),
                                         q2 = quant1(v[j].z, inv, stat), q3 = quant1(v[j].w, inv, stat);
                    d[j * kThreads + threadIdx.x] = make_uint2(q0 | (unsigned)q1 << 16, q2 | (unsigned)q3 << 16);
                }
            } else {
                float4* d = reinterpret_cast<float4*>((float*)a.in[k].dst + base);
#pragma unroll
                for (int j = 0; j < kPerThread / 4; ++j) d[j * kThreads + threadIdx.x] = v[j];
            }
        } else {
            // the last chunk of a tensor, or an address that is not 16-byte aligned
            const long long end = left < kChunk ? left : kChunk;
#pragma unroll 4
            for (long long i = threadIdx.x; i < end; i += kThreads) {
                const float x = __ldcs(src + base + i);
                if (flex) ((short*)a.in[k].dst)[base + i] = quant1(x, inv, stat);
                else ((float*)a.in[k].dst)[base + i] = x;
            }
        }
    }
    if (a.n && a.in[cur].flex_slot >= 0) b2_block_stat(stat, stats + a.in[cur].flex_slot, ismem);
}

// chunks of the inputs, and the launch: values a thread takes by how much there is in all
cudaError_t launch_inputs(Inputs& a, const b2_call_block* block, b2_flex_scale* table, int* stats, cudaStream_t st) {
    long long chunks = 0, total = 0;
    for (int i = 0; i < a.n; ++i) total += a.in[i].n;
    const bool brief = total < 148LL * 2 * kThreads * kPerLong;
    const int kChunk = kThreads * (brief ? kPerShort : kPerLong);
    for (int i = 0; i < a.n; ++i) {
        a.first_chunk[i] = chunks;
        chunks += (a.in[i].n + kChunk - 1) / kChunk;
    }
    a.first_chunk[a.n] = chunks;
    const unsigned grid = (unsigned)(chunks < 1 ? 1 : chunks > 148 * 8 ? 148 * 8 : chunks);
    if (brief) k_call_inputs<kPerShort><<<grid, kThreads, 0, st>>>(a, block, table, stats);
    else k_call_inputs<kPerLong><<<grid, kThreads, 0, st>>>(a, block, table, stats);
    return cudaGetLastError();
}

// Words alone: few parameters, which the host writes sooner (333 x 1001 values from another device tensor in every call
// 26.3 us with the launch above, 25.7 with this one, 22.8 where the word holds the address already).
struct Words {
    static constexpr int kMost = 4;
    int n;
    const void** where[kMost];
    const void* address[kMost];
};
__global__ void k_call_words(const Words w) {
    if (threadIdx.x < w.n) *w.where[threadIdx.x] = w.address[threadIdx.x];
}

struct Outputs {
    int n;
    b2_call_output out[B2_CALL_MAX_OUTPUTS];
    int first_block[B2_CALL_MAX_OUTPUTS + 1];
};

// End of a call: results, flex statistics and status word into pinned host memory the device can
// address, statistics cleared.  Block 0 takes statistics and status, the others 4 KB of a result each:
// bound by one read and one posted write over PCIe (blocks that went through the results one after another
// waited for every read: five results and ten blocks 6.9 -> 5.1 us, seven blocks 7.2 -> 4.0 us).
__global__ void __launch_bounds__(kThreads)
k_call_outputs(const Outputs o, int* __restrict__ stats, int n_stats, const int* __restrict__ status,
               int* __restrict__ host_stats, int* __restrict__ host_status) {
    after_earlier_kernels();
    if (blockIdx.x == 0) {
        const int word = threadIdx.x == 0 && status ? *status : 0;
        for (int i = threadIdx.x; i < n_stats; i += kThreads) {
            host_stats[i] = stats[i];
            stats[i] = 0;
        }
        if (threadIdx.x == 0 && status) *host_status = word;
    } else {
        int k = 0;
        while ((int)blockIdx.x - 1 >= o.first_block[k + 1]) ++k;
        const long long at = ((long long)((int)blockIdx.x - 1 - o.first_block[k]) * kThreads + threadIdx.x) * 16;
        const long long left = o.out[k].bytes - at;
        const char* s = (const char*)o.out[k].src + at;       // (allocations are 16-byte aligned)
        char* d = (char*)o.out[k].dst + at;
        if (left >= 16) *reinterpret_cast<uint4*>(d) = *reinterpret_cast<const uint4*>(s);
        else
            for (int i = 0; i < left; i += 2)                  // (elements are 2 or 4 bytes)
                *(unsigned short*)(d + i) = *(const unsigned short*)(s + i);
    }
}

#if defined(__x86_64__)
// Pageable memory to the pinned block: streaming stores, so that the lines the GPU is about to read
// are not first fetched and then left dirty in the cache.
__attribute__((target("avx2"))) void copy_streaming(void* dst, const void* src, size_t n) {
    char* d = (char*)dst;
    const char* s = (const char*)src;
    size_t i = 0;
    for (; i + 128 <= n; i += 128) {
        const __m256i a = _mm256_loadu_si256((const __m256i*)(s + i));
        const __m256i b = _mm256_loadu_si256((const __m256i*)(s + i + 32));
        const __m256i c = _mm256_loadu_si256((const __m256i*)(s + i + 64));
        const __m256i e = _mm256_loadu_si256((const __m256i*)(s + i + 96));
        _mm256_stream_si256((__m256i*)(d + i), a);
        _mm256_stream_si256((__m256i*)(d + i + 32), b);
        _mm256_stream_si256((__m256i*)(d + i + 64), c);
        _mm256_stream_si256((__m256i*)(d + i + 96), e);
    }
    if (i < n) memcpy(d + i, s + i, n - i);
    _mm_sfence();
}
#endif

// largest dec in [0, 31] with a * 2^dec <= 32767; -1 for a <= 0
int largest_dec(double a) {
    if (!(a > 0.0)) return -1;
    if (std::isinf(a)) return 0;
    int e;
    (void)std::frexp(a, &e);
    int dec = 15 - e;
    if (std::ldexp(a, dec + 1) <= 32767.0) dec += 1;
    while (std::ldexp(a, dec) > 32767.0) dec -= 1;
    return dec < 0 ? 0 : dec > 31 ? 31 : dec;
}

}  // namespace

extern "C" int b2_call_inputs(const b2_call_input* inputs, int32_t n, const b2_call_block* block,
                              b2_flex_scale* table, int32_t* stats, void* stream) {
    static_assert(sizeof(b2_call_arg) == 16 && offsetof(b2_call_block, arg) % 16 == 0, "read as one word");
    B2_REQUIRE(n >= 0 && n <= B2_CALL_MAX_INPUTS && (n == 0 || inputs) && block &&
               ((uintptr_t)block & 15) == 0, "bad argument");
    Inputs a = {};
    a.n = n;
    for (int i = 0; i < n; ++i) {
        B2_REQUIRE(inputs[i].dst && inputs[i].n >= 0 && (inputs[i].flex_slot < 0 || stats), "bad argument");
        a.in[i] = inputs[i];
    }
    B2_CUDA(launch_inputs(a, block, table, stats, (cudaStream_t)stream));
    return B2_OK;
}

namespace {
void copy_to_pinned(void* pinned, const void* src, size_t bytes) {
#if defined(__x86_64__)
    static const bool avx2 = __builtin_cpu_supports("avx2");
    if (avx2 && ((uintptr_t)pinned & 31) == 0) return copy_streaming(pinned, src, bytes);
#endif
    memcpy(pinned, src, bytes);
}
}  // namespace

extern "C" int b2_call_take(const b2_call_input* inputs, int32_t n, const b2_call_block* block,
                            const void* const* pageable, b2_flex_scale* table, int32_t* stats, int32_t* launches,
                            int32_t device, void* stream) {
    B2_REQUIRE(n >= 0 && n <= B2_CALL_MAX_INPUTS && (n == 0 || inputs) && block && launches, "bad argument");
    B2_REQUIRE(block->table_rows <= 0 || (table && block->table), "rows without a table");
    *launches = 0;
    int current = device;
    B2_CUDA(cudaGetDevice(&current));
    const struct Back {                                        // (stream 0 is the current device's)
        int to, from;
        Back(int t, int f) : to(t), from(f) { if (to != from) cudaSetDevice(from); }
        ~Back() { if (to != from) cudaSetDevice(to); }
    } back(current, device);
    // A piece of pageable memory: the host copies about 20 GB/s and a launch costs it 2 us, PCIe brings
    // 50 GB/s: less than 192 KB (10 us of copying, 4 of reading) is not worth another launch.
    const long long least = 48 << 10;                          // values
    Inputs a = {};
    const void** holds[B2_CALL_MAX_INPUTS];
    a.rows = block->table;
    a.n_rows = block->table_rows > 0 ? block->table_rows : 0;
    for (int k = 0; k < n; ++k) {
        B2_REQUIRE(inputs[k].dst && inputs[k].n >= 0 && (inputs[k].flex_slot < 0 || stats), "bad argument");
        const void* src = block->arg[k].src;
        if (!inputs[k].where) continue;
        // (where there is nothing to copy the values are in their place)
        const void* address = src && block->arg[k].in_place ? src : inputs[k].dst;
        if (inputs[k].holds) {
            if (*inputs[k].holds == address) continue;
            *inputs[k].holds = nullptr;                        // (until the launch is on its way)
        }
        a.where[a.n_words] = inputs[k].where;
        a.address[a.n_words] = address;
        holds[a.n_words++] = inputs[k].holds;
    }
    auto add = [&](const b2_call_input& in, const b2_call_arg& arg, long long first, long long count) {
        a.in[a.n] = in;
        a.in[a.n].n = count;
        a.in[a.n].dst = (char*)in.dst + first * (in.flex_slot >= 0 ? 2 : 4);
        a.src[a.n] = (const float*)arg.src + first;
        a.inv[a.n++] = arg.inv_scale;
    };
    auto launch = [&]() -> cudaError_t {
        cudaError_t e;
        if (a.n || a.n_rows || a.n_words > Words::kMost) {
            e = launch_inputs(a, nullptr, table, stats, (cudaStream_t)stream);
        } else {
            Words w = {a.n_words};
            for (int i = 0; i < w.n; ++i) { w.where[i] = a.where[i]; w.address[i] = a.address[i]; }
            k_call_words<<<1, 32, 0, (cudaStream_t)stream>>>(w);
            e = cudaGetLastError();
        }
        ++*launches;
        for (int i = 0; i < a.n_words && e == cudaSuccess; ++i)
            if (holds[i]) *holds[i] = a.address[i];
        a.n = a.n_words = a.n_rows = 0;
        return e;
    };
    for (int pass = 0; pass < 2; ++pass)                       // pageable memory last
        for (int k = 0; k < n; ++k) {
            const b2_call_arg& arg = block->arg[k];
            const bool staged = pageable && pageable[k];
            if (!arg.src || (arg.in_place && inputs[k].where) || staged != (pass == 1)) continue;
            if (!staged) { add(inputs[k], arg, 0, inputs[k].n); continue; }
            const long long count = inputs[k].n;
            long long piece = count / 4 / 4096 * 4096;
            if (piece < least) piece = least;
            for (long long at = 0; at < count; at += piece) {
                const long long now = count - at < piece + piece / 2 ? count - at : piece;
                copy_to_pinned((float*)arg.src + at, (const float*)pageable[k] + at, (size_t)now * 4);
                add(inputs[k], arg, at, now);
                if (at + now < count) { B2_CUDA(launch()); continue; }
                break;
            }
        }
    if (a.n || a.n_words || a.n_rows) B2_CUDA(launch());
    return B2_OK;
}

extern "C" int b2_call_outputs(const b2_call_output* outputs, int32_t n, int32_t* stats,
                               int32_t n_stats, const int32_t* status, int32_t* host_stats,
                               int32_t* host_status, void* stream) {
    B2_REQUIRE(n >= 0 && n <= B2_CALL_MAX_OUTPUTS && (n == 0 || outputs), "bad argument");
    B2_REQUIRE(n_stats >= 0 && (n_stats == 0 || (stats && host_stats)), "bad argument");
    B2_REQUIRE((status == nullptr) == (host_status == nullptr), "status source and destination go together");
    Outputs o;
    o.n = n;
    o.first_block[0] = 0;
    for (int i = 0; i < n; ++i) {
        B2_REQUIRE(outputs[i].src && outputs[i].dst && outputs[i].bytes >= 0 &&
                   (((uintptr_t)outputs[i].src | (uintptr_t)outputs[i].dst) & 15) == 0,
                   "results must be 16-byte aligned");
        const long long blocks = (outputs[i].bytes + kThreads * 16 - 1) / (kThreads * 16);
        B2_REQUIRE(o.first_block[i] + blocks < (1 << 30), "results too large");
        o.out[i] = outputs[i];
        o.first_block[i + 1] = o.first_block[i] + (int)blocks;
    }
    const int grid = 1 + o.first_block[n];
    B2_CUDA(b2::launch_after(k_call_outputs, dim3((unsigned)grid), kThreads, 0, (cudaStream_t)stream, o, stats, n_stats, status,
                                                                          host_stats, host_status));
    B2_CUDA(cudaGetLastError());
    return B2_OK;
}

extern "C" int b2_call_wait(int32_t device, void* stream) {
    int current = device;
    B2_CUDA(cudaGetDevice(&current));
    if (current != device) B2_CUDA(cudaSetDevice(device));         // (stream 0 is the current device's)
    const cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
    if (current != device) cudaSetDevice(current);
    B2_CUDA(e);
    return B2_OK;
}

extern "C" int b2_call_stage(const void* src, size_t bytes, void* pinned, const void** visible) {
    B2_REQUIRE(src && visible, "null argument");
    cudaPointerAttributes at;
    const cudaError_t e = cudaPointerGetAttributes(&at, src);
    if (e == cudaSuccess && at.type == cudaMemoryTypeHost && at.devicePointer) {
        *visible = at.devicePointer;              // page-locked: the kernel reads it where it is
        return B2_OK;
    }
    (void)cudaGetLastError();                     // (not a CUDA address: no error of the caller's)
    *visible = nullptr;
    if (!pinned) return B2_OK;                    // pageable, and no block to copy to
    copy_to_pinned(pinned, src, bytes);
    *visible = pinned;
    return B2_OK;
}

static int set_row(int64_t slot, int64_t dec, int64_t* uploaded, b2_flex_scale* host_table) {
    if (uploaded[slot] == dec) return 0;
    uploaded[slot] = dec;
    host_table[slot].scale = std::ldexp(1.0f, (int)-dec);
    host_table[slot].inv_scale = std::ldexp(1.0f, (int)dec);
    return 1;
}

extern "C" int b2_flex_begin_call(const b2_flex_state* s, int32_t n, const int64_t* ids,
                                  const int64_t* slot_write, const int64_t* slot_read,
                                  int64_t* uploaded, b2_flex_scale* host_table, int32_t* changed) {
    B2_REQUIRE(s && n >= 0 && (n == 0 || (ids && slot_write && slot_read)) && uploaded && host_table &&
               changed, "null argument");
    int ch = 0;
    auto row = [&](int64_t slot, int64_t dec) { ch |= set_row(slot, dec, uploaded, host_table); };
    for (int32_t k = 0; k < n; ++k) {
        const int64_t i = ids[k], stored = s->dec[i];
        if (s->initialized[i] && s->pending[i] >= 0) {
            s->dec[i] = s->pending[i];
            s->pending[i] = -1;
        }
        row(slot_write[k], s->dec[i]);
        if (slot_read[k] != slot_write[k]) row(slot_read[k], stored);
    }
    *changed = ch;
    return B2_OK;
}

extern "C" int b2_flex_rows_written(const b2_flex_state* s, int32_t n, const int64_t* ids, const int64_t* slot_read,
                                    int64_t* uploaded, b2_flex_scale* host_table, int32_t* changed) {
    B2_REQUIRE(s && n >= 0 && (n == 0 || (ids && slot_read)) && uploaded && host_table && changed, "null argument");
    int ch = 0;
    for (int32_t k = 0; k < n; ++k) ch |= set_row(slot_read[k], s->dec[ids[k]], uploaded, host_table);
    *changed = ch;
    return B2_OK;
}

extern "C" int b2_flex_end_call(const b2_flex_state* s, int32_t n, const int64_t* ids,
                                const int64_t* slots, const int32_t* maxima, int32_t* undecided,
                                int32_t* n_undecided, int32_t* settled) {
    B2_REQUIRE(s && n >= 0 && (n == 0 || (ids && maxima && undecided)) && n_undecided && settled,
               "null argument");
    const int H = B2_FLEX_HISTORY;
    int open = 0, all = 1;
    for (int32_t k = 0; k < n; ++k) {
        const int64_t i = ids[k];
        const int64_t m = maxima[slots ? slots[k] : k];
        const double scale = std::ldexp(1.0, (int)-s->dec[i]);
        auto push = [&](double v) {
            int64_t& pos = s->hist_pos[i];
            s->hist[i * H + pos] = v;
            pos = (pos + 1) % H;
            if (s->hist_len[i] < H) s->hist_len[i] += 1;
        };
        if (m >= 32767) {
            s->overflows[i] += 1;
            s->run_length[i] = 0;
            push(2.0 * (double)m * scale);
            s->pending[i] = s->dec[i] - 2 < 0 ? 0 : s->dec[i] - 2;
            all = 0;
            continue;
        }
        const double value = (double)m * scale;
        if (value == s->run_value[i]) {
            s->run_length[i] += 1;
            if (s->run_length[i] > H) {
                // the window already holds nothing but this value: the same choice as before
                s->pending[i] = s->run_choice[i];
                if (s->pending[i] >= 0 && s->pending[i] != s->dec[i]) all = 0;
                continue;
            }
        } else {
            s->run_value[i] = value;
            s->run_length[i] = 1;
        }
        all = 0;
        push(value);
        const double* h = s->hist + i * H;
        const int len = (int)s->hist_len[i];
        double sum = 0.0, var = 0.0, top = h[0];
        for (int j = 0; j < len; ++j) { sum += h[j]; if (h[j] > top) top = h[j]; }
        const double mean = sum / len;
        for (int j = 0; j < len; ++j) var += (h[j] - mean) * (h[j] - mean);
        const double predicted = top + 3.0 * std::sqrt(var / len);
        const int choice = largest_dec(predicted);
        // these sums are not the exactly rounded ones of the rule: where the value lies within a
        // hair of the point at which the choice changes, the caller decides with exact sums
        if (choice >= 0 && !std::isinf(predicted) &&
            (std::fabs(std::ldexp(predicted, choice) - 32767.0) < 1e-6 * 32767.0 ||
             std::fabs(std::ldexp(predicted, choice + 1) - 32767.0) < 1e-6 * 32767.0))
            undecided[open++] = k;
        s->pending[i] = choice;
        s->run_choice[i] = choice;
    }
    *n_undecided = open;
    *settled = all;
    return B2_OK;
}
