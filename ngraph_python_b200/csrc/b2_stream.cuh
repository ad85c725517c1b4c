// Matrix product in one launch: C[M,N] = A[M,K] * B[N,K]^T with the operands converted on the way in, for
// problems where the pre-pass of the plane kernels (b2_gemm_impl.cuh) and its launches cost as much as the
// product.
//
// One CTA per 128 x BN tile (times a slice of K), 800 threads:
//   eight warps copy: k-blocks of both operands as they lie into a ring of raw stages, sixteen bytes to a cp.async
//             whatever a line's alignment (it keeps its place within sixteen bytes, and who reads it shifts); in groups
//             that take the k-blocks by turns where there are several;
//   four groups of four warps convert, the k-blocks by turns: A's two planes go to tensor memory (a lane is a
//             row), B's K-major and 128-byte swizzled to shared memory; afterwards all sixteen are the epilogue;
//   one warp: tensor memory, tcgen05.mma with A from tensor memory.
// A k-block is 128 bytes of plane: 32 fp32 or 128 int16 values.
//   fp32:   3xTF32, chains of 16 k-blocks (the tensor core's fp32 sum truncates), each with a sum of its own in
//           tensor memory, added to nearest in the order of the chains -- what the other product kernels do, so that
//           the same rows and columns give the same bits whichever takes them (a mask `x > 0` of a value near
//           zero would otherwise change with the dispatch).
//   flex16: four exact int8 products, HH | X | LL as in b2_gemm_impl.cuh.
// Slices of K: the CTAs of a cluster (up to 8) take one each; their sums meet in distributed shared memory, where
// every CTA adds a share of the columns in the order of the slices and finishes them.
//
// What bounds it: latency at the smallest sizes, then shared memory's 128 bytes a clock.  An instruction of few
// columns reads 4 KB of A from shared memory in 39 cycles and writes next to nothing; from tensor memory it takes 9
// (N = 16) to 64 (N = 128, the tensor pipe's own rate).  A k-block then takes 370 + 9 BN (fp32) or 900 + 16 BN
// (flex16) cycles, which is instruction issue: copies, conversion and the issue of its twelve or sixteen MMAs.  One
// B200, the kernel of b2_direct.cuh -> this one, us: fp32 512 x 128 x 512 10.7 -> 8.6, by columns 13.6 -> 10.0; flex16
// 512 x 128 x 784 8.8 -> 7.6, 300 x 50 x 300 9.6 -> 6.5, 187 x 131 x 31 12.4 -> 6.8 (a result is a chain of a hundred
// dependent instructions: one to four of them to a thread instead of eight, loads without branches between them).
#ifndef B2_STREAM_CUH
#define B2_STREAM_CUH
#include "b2_direct.h"
#include "b2_gemm_impl.cuh"

namespace {

constexpr int kStrThreads = 800;
constexpr int kStrCopy = 512;              // first copying thread; the MMA warp is the last
constexpr int kStrGroups = 4;              // of converters
// planes of k-blocks under way: 64 columns of tensor memory each
__host__ __device__ constexpr int str_slots(int bn) { return bn == 128 ? 2 : 4; }

struct StreamParams {
    b2_direct_args a;
    int num_kb, kb_per_split, splits, chains, stages, tmem;
};

// A raw stage holds lines -- rows of a k-block where K is contiguous, else columns -- sixteen bytes longer than what
// they hold: room for their place within sixteen, and neighbours' chunks in different banks.
__host__ __device__ constexpr int str_line(int mode, int rows, int kind) {
    return (kind == B2_OPERAND_K ? (mode == MODE_FLEX16 ? 256 : 128) : rows * (mode == MODE_FLEX16 ? 2 : 4)) + 16;
}
__host__ __device__ constexpr int str_operand_bytes(int mode, int rows, int kind) {
    return str_line(mode, rows, kind) * (kind == B2_OPERAND_K ? rows : mode == MODE_FLEX16 ? 128 : 32);
}
__host__ __device__ constexpr int str_raw_bytes(int mode, int bn, int ak, int bk) {
    return str_operand_bytes(mode, 128, ak) + str_operand_bytes(mode, bn, bk);
}
__host__ __device__ constexpr int str_plane_bytes(int bn) { return 2 * bn * 128; }
__host__ __device__ constexpr int str_most_stages(int mode, int bn) {
    return mode == MODE_FLEX16 ? (bn <= 32 ? 4 : bn == 64 ? 3 : 2) : (bn <= 32 ? 7 : bn == 64 ? 5 : 4);
}

// ---- copies -----------------------------------------------------------------------------------------
// sixteen bytes of shared memory <- `valid` bytes at src, then zeros (no byte is read where that is 0)
__device__ __forceinline__ void cp_async16(unsigned dst, const void* src, int valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
}
// this thread's arrival at the barrier, once all its copies so far have landed
__device__ __forceinline__ void cp_async_arrive(unsigned long long* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ int within16(int n) { return n < 0 ? 0 : n > 16 ? 16 : n; }
// A thread's chunks of an operand's k-blocks: of lines STEP apart, the same place in each.
template <int MODE, int ROWS, int KIND, int THREADS>
struct ChunkWalk {
    static constexpr int ES = MODE == MODE_FLEX16 ? 2 : 4, KB = MODE == MODE_FLEX16 ? 128 : 32;
    static constexpr int LINE = str_line(MODE, ROWS, KIND), ALONG = (LINE - 16) / 16;           // chunks of a line
    static constexpr int LINES = KIND == B2_OPERAND_K ? ROWS : KB;
    static constexpr int COUNT = (LINES * ALONG + THREADS - 1) / THREADS;
    static constexpr int STEP = THREADS / ALONG;
    static constexpr bool PART = LINES * ALONG % THREADS != 0;         // not every thread has its last chunk
    const char* first;                     // line 0 of this k-block
    long long line_bytes, kb_step;
    int line, c, ct;
    int there;                             // K contiguous: lines that exist; else the bytes of a line that do

    __device__ __forceinline__ ChunkWalk(const void* base, long long rs, long long ks, int row0, int rows_all, int k0, int t,
                                         int kb_apart) {
        ct = t;
        line = ct / ALONG;
        c = ct % ALONG;
        first = (const char*)base + (KIND == B2_OPERAND_K ? (long long)row0 * rs + k0 : (long long)k0 * ks + row0) * ES;
        line_bytes = (KIND == B2_OPERAND_K ? rs : ks) * ES;
        kb_step = (KIND == B2_OPERAND_K ? ES : ks * ES) * KB * kb_apart;
        const int rows = rows_all - row0;
        there = KIND == B2_OPERAND_K ? rows : (rows > ROWS ? ROWS : rows) * ES;
    }
    // bytes of a line that exist; `left`: columns from the k-block's first to the end of K, at most KB
    __device__ __forceinline__ int bytes(int l, int left) const {
        if (KIND == B2_OPERAND_K) return l < there ? left * ES : 0;
        return l < left ? there : 0;
    }
    // one k-block; the next call takes the one `kb_apart` behind it
    template <bool EVEN>
    __device__ __forceinline__ void bring(unsigned char* raw, int left) {
        const unsigned to = smem_u32(raw) + line * LINE + c * 16;
        left = left < KB ? left : KB;
        const char* p = first + line * line_bytes;
        const long long step = STEP * line_bytes;
        if (EVEN) {
            p += c * 16;
            // (all k-blocks but the last: nothing to work out)
            const bool full = left == KB;
            const int n_full = KIND == B2_OPERAND_K ? 16 : within16(there - 16 * c);
            if (full) {
#pragma unroll (COUNT < 8 ? COUNT : 8)
                for (int i = 0; i < COUNT; ++i, p += step) {
                    if (PART && line + i * STEP >= LINES) break;
                    cp_async16(to + i * STEP * LINE, p, KIND != B2_OPERAND_K || line + i * STEP < there ? n_full : 0);
                }
            } else {
#pragma unroll 2
                for (int i = 0; i < COUNT; ++i, p += step) {
                    if (PART && line + i * STEP >= LINES) break;
                    cp_async16(to + i * STEP * LINE, p, within16(bytes(line + i * STEP, left) - 16 * c));
                }
            }
        } else {
            // The sixteen bytes that a line starts in are read from their beginning: what stands in front of it is not
            // used, and an aligned chunk that holds a byte of the operand does not cross a page.
#pragma unroll (COUNT < 8 ? COUNT : 8)
            for (int i = 0; i < COUNT; ++i, p += step) {
                if (PART && line + i * STEP >= LINES) break;
                const int d = (int)(uintptr_t)p & 15, n = bytes(line + i * STEP, left);
                cp_async16(to + i * STEP * LINE, p - d + 16 * c, n ? within16(d + n - 16 * c) : 0);
            }
            p = first + ct * line_bytes;
            for (int l = ct; l < LINES; l += THREADS, p += THREADS * line_bytes) {
                const int d = (int)(uintptr_t)p & 15, n = within16(d + bytes(l, left) - 16 * ALONG);
                if (d) cp_async16(smem_u32(raw) + l * LINE + ALONG * 16, p - d + 16 * ALONG, n);
            }
        }
        first += kb_step;
    }
};

// ---- conversion -------------------------------------------------------------------------------------
// a = hi + lo with hi rounded to tf32, ties away from zero: what cvt.rna.tf32 gives for every finite a
// (infinities and NaN end as NaN in the product either way), on the full-rate integer pipe
__device__ __forceinline__ void str_split_tf32(unsigned a, unsigned& hi, unsigned& lo) {
    hi = (a + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(__uint_as_float(a) - __uint_as_float(hi));
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// four consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tmem_ld4(unsigned taddr, unsigned* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
template <int MODE>
__device__ __forceinline__ void tc_mma_ta(unsigned tmem_d, unsigned tmem_a, unsigned long long bdesc, unsigned idesc,
                                          unsigned accumulate) {
    if (MODE == MODE_FLEX16)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// N words at `at` + d bytes, 16-byte aligned but for d
template <int MODE, int N>
__device__ __forceinline__ void raw_words(const unsigned char* at, int d, unsigned* v) {
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
        const uint4 t = ((const uint4*)at)[q];
        v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
    }
    if (d == 0) return;
    const uint4 t = ((const uint4*)at)[N / 4];
    unsigned w[5] = {t.x, t.y, t.z, t.w, 0u};
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = d & 8 ? (j + 2 < N ? v[j + 2] : w[j + 2 - N]) : v[j];
    if (d & 8) { w[0] = w[2]; w[1] = w[3]; }
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = d & 4 ? (j + 1 < N ? v[j + 1] : w[0]) : v[j];
    if (d & 4) w[0] = w[1];
    if (MODE == MODE_FLEX16) {
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = d & 2 ? __funnelshift_r(v[j], j + 1 < N ? v[j + 1] : w[0], 16) : v[j];
    }
}
// Words [from, from + N) of what is to be a row of planes (a word: one fp32 or two int16 columns), from a raw stage.
// `place`: where the operand's first line lies within sixteen bytes, `apart` how far apart lines are (modulo 16).
template <int MODE, int ROWS, int KIND, int N>
__device__ __forceinline__ void raw_row(const unsigned char* raw, int row, int from, int place, int apart, unsigned* v) {
    constexpr int LINE = str_line(MODE, ROWS, KIND);
    if (KIND == B2_OPERAND_K) {
        raw_words<MODE, N>(raw + row * LINE + from * 4, (place + row * apart) & 15, v);
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            if (MODE != MODE_FLEX16) {
                const int k = from + j;
                v[j] = *(const unsigned*)(raw + k * LINE + ((place + k * apart) & 15) + row * 4);
            } else {
                const int k = 2 * (from + j);
                v[j] = (unsigned)*(const unsigned short*)(raw + k * LINE + ((place + k * apart) & 15) + row * 2) |
                       (unsigned)*(const unsigned short*)(raw + (k + 1) * LINE + ((place + (k + 1) * apart) & 15) + row * 2) << 16;
            }
        }
    }
}
// N words of both planes from N (fp32) or 2N (flex16) words
template <int MODE, int N>
__device__ __forceinline__ void to_planes(const unsigned* v, unsigned* hi, unsigned* lo) {
#pragma unroll
    for (int j = 0; j < N; ++j) {
        if (MODE != MODE_FLEX16) {
            str_split_tf32(v[j], hi[j], lo[j]);
        } else {
            hi[j] = __byte_perm(v[2 * j], v[2 * j + 1], 0x7531);
            lo[j] = __byte_perm(v[2 * j], v[2 * j + 1], 0x6420);
        }
    }
}
template <int W>
__device__ __forceinline__ void tmem_st(unsigned taddr, const unsigned* r) {
    if (W == 8) asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
    else asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[W - 8]),
          "r"(r[W - 7]), "r"(r[W - 6]), "r"(r[W - 5]), "r"(r[W - 4]), "r"(r[W - 3]), "r"(r[W - 2]), "r"(r[W - 1]) : "memory");
}

// EVEN: all lines of both operands start on sixteen bytes
template <int MODE, int BN, int AK, int BK, bool EVEN>
__global__ void __launch_bounds__(kStrThreads, 1)
stream_kernel(const __grid_constant__ StreamParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr bool FLEX = MODE == MODE_FLEX16;
    constexpr int KB = FLEX ? 128 : 32, RAW = str_raw_bytes(MODE, BN, AK, BK), PLANES = str_plane_bytes(BN);
    constexpr int A_RAW = str_operand_bytes(MODE, 128, AK), ES = FLEX ? 2 : 4;
    constexpr int kMost = str_most_stages(MODE, BN), SLOTS = str_slots(BN);
    // groups of copying warps: a k-block costs each of their threads a chain of some hundred cycles beside the copies
    constexpr int COPY_GROUPS = FLEX ? 2 : 4;
    typedef typename std::conditional<FLEX, long long, float>::type Sum;
    unsigned char* planes = smem;                                                 // [slots][hi, lo][BN][128]
    unsigned char* ring = smem + SLOTS * PLANES;                                  // [stages][A | B]
    __shared__ unsigned long long raw_full[kStrGroups][kMost], raw_empty[kStrGroups][kMost], slot_full[kStrGroups], slot_empty[kStrGroups], sums_full;
    __shared__ unsigned tmem_holder;
    __shared__ int fail_flag;

    const int wid = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const b2_direct_args& a = p.a;
    const int m0 = blockIdx.y * 128, n0 = blockIdx.x * BN;
    const int rank = blockIdx.z, kb0 = rank * p.kb_per_split;
    const int nkb = min(p.kb_per_split, p.num_kb - kb0), stages = p.stages;
    const int copy_groups = nkb >= COPY_GROUPS ? COPY_GROUPS : 1;

    if (threadIdx.x < kMost * kStrGroups) {
        // (a stage's barriers per group that waits at them: a waiter must see every phase in turn, a parity does not
        // tell phase n from phase n+2)
        mbar_init(&raw_full[0][0] + threadIdx.x, 256 / copy_groups);
        mbar_init(&raw_empty[0][0] + threadIdx.x, 4);
        if (threadIdx.x < kStrGroups) {
            mbar_init(&slot_full[threadIdx.x], 4);
            mbar_init(&slot_empty[threadIdx.x], 1);
        }
        if (threadIdx.x == 0) {
            mbar_init(&sums_full, 1);
            fail_flag = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (wid == 24) {
        tmem_alloc(&tmem_holder, p.tmem);
        // the next kernel may start its set-up now: not before this CTA holds its tensor memory, or
        // the two could each wait for what the other has
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = (unsigned)warp_uniform((int)tmem_holder);
    const unsigned tmem_sums = tmem_base + SLOTS * 64;
    float scale_a = 1.0f, scale_b = 1.0f, step_c = 1.0f;
    // everything before this line touches no global memory; everything after it sees the completed work of
    // all earlier kernels of the stream
    if (wid >= 16 && wid < 24) {
        // ---- copies
        auto copies = [&](auto groups) {
            constexpr int GROUPS = decltype(groups)::value, THREADS = 256 / GROUPS;
            const int cg = (wid - 16) / (8 / GROUPS), ct = ((int)threadIdx.x - kStrCopy) % THREADS;
            ChunkWalk<MODE, 128, AK, THREADS> wa(a.A, a.a_rs, a.a_ks, m0, a.M, (kb0 + cg) * KB, ct, GROUPS);
            ChunkWalk<MODE, BN, BK, THREADS> wb(a.B, a.b_rs, a.b_ks, n0, a.N, (kb0 + cg) * KB, ct, GROUPS);
            asm volatile("griddepcontrol.wait;" ::: "memory");
            bool ok = true;
            int s = cg % stages, left = a.K - (kb0 + cg) * KB;
            unsigned bits = 0;                                  // (bit s: parity of the next phase of stage s)
            for (int kb = cg; kb < nkb; kb += GROUPS) {
                if (ok && kb >= stages) {
                    if (!mbar_wait(&raw_empty[cg][s], (bits >> s) & 1u)) { atomicExch(&fail_flag, 1); ok = false; }
                    bits ^= 1u << s;
                }
                unsigned char* raw = ring + s * RAW;
                wa.template bring<EVEN>(raw, left);
                wb.template bring<EVEN>(raw + A_RAW, left);
                cp_async_arrive(&raw_full[kb % kStrGroups][s]);
                left -= GROUPS * KB;
                s += GROUPS;
                while (s >= stages) s -= stages;
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        };
        if (copy_groups > 1) copies(std::integral_constant<int, COPY_GROUPS>());
        else copies(std::integral_constant<int, 1>());
    } else if (wid < 16) {
        // ---- converters
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (FLEX && !a.probe) {                                 // (while the first k-blocks are on their way)
            scale_a = __ldcg(&a.table[a.slotA].scale);
            scale_b = __ldcg(&a.table[a.slotB].scale);
            step_c = __ldcg(&a.table[a.slotC].inv_scale);
        }
        const int group = wid >> 2, quarter = wid & 3;
        const int row = quarter * 32 + lane, t = quarter * 32 + lane;
        constexpr int UNITS = BN * 8, PER = UNITS / 128;        // chunks of B, of a thread
        auto b_row = [&](int u) { return BK == B2_OPERAND_K ? u >> 3 : u % BN; };      // neighbouring lanes: chunks of a
        auto b_chunk = [&](int u) { return BK == B2_OPERAND_K ? u & 7 : u / BN; };     // row, or rows
        // where lines stand within sixteen bytes: the same in every k-block (KB lines or columns are a multiple of that)
        const int a_apart = EVEN ? 0 : (int)((AK == B2_OPERAND_K ? a.a_rs : a.a_ks) * ES & 15), b_apart = EVEN ? 0 : (int)((BK == B2_OPERAND_K ? a.b_rs : a.b_ks) * ES & 15);
        const int a_place = EVEN ? 0 : ((int)(uintptr_t)a.A & 15) + (AK == B2_OPERAND_K ? m0 * a_apart : m0 * ES) & 15;
        const int b_place = EVEN ? 0 : ((int)(uintptr_t)a.B & 15) + (BK == B2_OPERAND_K ? n0 * b_apart : n0 * ES) & 15;
        bool ok = true;
        int s = group % stages;
        unsigned raw_bits = 0, slot_parity = 1;                 // (bit s as above)
        for (int kb = group; kb < nkb; kb += kStrGroups) {
            const int slot = kb % SLOTS;
            const unsigned slot_a = tmem_base + slot * 64 + ((unsigned)(quarter * 32) << 16);
            unsigned char* bp = planes + slot * PLANES;
            if (ok && !mbar_wait(&raw_full[group][s], (raw_bits >> s) & 1u)) { atomicExch(&fail_flag, 1); ok = false; }
            raw_bits ^= 1u << s;
            const unsigned char* raw = ring + s * RAW;
            // so many words of both planes at a time
            constexpr int W = EVEN && !FLEX ? 16 : 8, FROM = FLEX ? 2 : 1;
            unsigned v[W * FROM], hi[W], lo[W];
            constexpr bool FIRST = EVEN && !FLEX;               // (read while the slot is still in use)
            if (FIRST) {
                raw_row<MODE, 128, AK, W * FROM>(raw, row, 0, a_place, a_apart, v);
                to_planes<MODE, W>(v, hi, lo);
            }
            if (kb >= SLOTS) {
                slot_parity ^= 1u;
                if (ok && !mbar_wait(&slot_empty[group], slot_parity)) { atomicExch(&fail_flag, 1); ok = false; }
                tc_fence_after();
            }
#pragma unroll (FLEX ? 1 : 32 / W)
            for (int q = 0; q < 32 / W; ++q) {
                if (!FIRST || q > 0) {
                    raw_row<MODE, 128, AK, W * FROM>(raw, row, q * W * FROM, a_place, a_apart, v);
                    to_planes<MODE, W>(v, hi, lo);
                }
                tmem_st<W>(slot_a + W * q, hi);
                tmem_st<W>(slot_a + 32 + W * q, lo);
            }
#pragma unroll (FLEX ? 1 : PER)
            for (int i = 0; i < PER; ++i) {
                const int u = t + 128 * i, at = b_row(u) * 128 + ((b_chunk(u) ^ (b_row(u) & 7)) << 4);
                raw_row<MODE, BN, BK, FLEX ? 8 : 4>(raw + A_RAW, b_row(u), b_chunk(u) * (FLEX ? 8 : 4), b_place, b_apart, v);
                to_planes<MODE, 4>(v, hi, lo);
                *(uint4*)(bp + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *(uint4*)(bp + BN * 128 + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            tmem_st_wait();
            tc_fence_before();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) { mbar_arrive(&slot_full[group]); mbar_arrive(&raw_empty[(kb + stages) % copy_groups][s]); }
            s += kStrGroups;
            while (s >= stages) s -= stages;
        }
    } else if (elect_one()) {
        // ---- MMA issue
        const unsigned id_ss = make_idesc(2, 1, 1, BN), id_su = make_idesc(2, 1, 0, BN),
                       id_us = make_idesc(2, 0, 1, BN), id_uu = make_idesc(2, 0, 0, BN), id_tf = make_idesc(1, 2, 2, BN);
        // (what an instruction needs stands in uniform registers: unrolled over the slots all of it is a constant away
        // from two bases, where it was worked out per k-block an instruction took 38 cycles)
        const unsigned long long desc = make_smem_desc(planes);
        unsigned sum = tmem_sums, parity = 0;
        bool ok = true;
        for (int kb4 = 0; kb4 < nkb && ok; kb4 += kStrGroups, parity ^= 1u) {
            if (!FLEX && kb4 > 0 && kb4 % kChunkKb == 0) sum += BN;
#pragma unroll
            for (int g = 0; g < kStrGroups; ++g) {
                if (kb4 + g >= nkb || !ok) break;
                if (!mbar_wait(&slot_full[g], parity)) { atomicExch(&fail_flag, 1); ok = false; break; }
                tc_fence_after();
                const unsigned ah = tmem_base + g % SLOTS * 64, al = ah + 32;
                const unsigned long long dB0 = desc + (g % SLOTS * PLANES >> 4), dB1 = dB0 + (BN * 128 >> 4);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const unsigned long long adv = (unsigned long long)(2 * k);
                    const unsigned acc = g > 0 || k > 0 || (FLEX ? kb4 : kb4 % kChunkKb) > 0 ? 1u : 0u;
                    if (FLEX) {
                        tc_mma_ta<MODE>(sum, ah + 8 * k, dB0 + adv, id_ss, acc);             // HH
                        tc_mma_ta<MODE>(sum + BN, ah + 8 * k, dB1 + adv, id_su, acc);        // X += ah*bl
                        tc_mma_ta<MODE>(sum + BN, al + 8 * k, dB0 + adv, id_us, 1u);         // X += al*bh
                        tc_mma_ta<MODE>(sum + 2 * BN, al + 8 * k, dB1 + adv, id_uu, acc);    // LL
                    } else if (a.colmajor) {
                        // (the order of the plane kernels, in terms of C's own operands)
                        tc_mma_ta<MODE>(sum, ah + 8 * k, dB0 + adv, id_tf, acc);             // hi*hi
                        tc_mma_ta<MODE>(sum, al + 8 * k, dB0 + adv, id_tf, 1u);
                        tc_mma_ta<MODE>(sum, ah + 8 * k, dB1 + adv, id_tf, 1u);
                    } else {
                        tc_mma_ta<MODE>(sum, ah + 8 * k, dB0 + adv, id_tf, acc);
                        tc_mma_ta<MODE>(sum, ah + 8 * k, dB1 + adv, id_tf, 1u);
                        tc_mma_ta<MODE>(sum, al + 8 * k, dB0 + adv, id_tf, 1u);
                    }
                }
                tc_commit(&slot_empty[(g + SLOTS) % kStrGroups]);         // of the group that fills the slot next
            }
        }
        tc_commit(&sums_full);
    }
    __syncwarp();

    // ---- epilogue: the sixteen converting warps; lane quarter = warp % 4, the four warps of a quarter share the
    // columns, few to a thread: a result costs a chain of a hundred dependent instructions or more
    const int quarter = wid & 3, part = wid >> 2;
    const int lrow = quarter * 32 + lane, row = m0 + lrow;
    const int splits = p.splits, chains = FLEX ? 1 : p.chains;
    Sum* red = (Sum*)smem;                                        // [chains][BN][128], slices only
    bool ok = true;
    int stat = 0, sh = 0;
    unsigned long long pmax = 0;
    unsigned rmask = 0, rhalf = 0;
    bool fast = false;
    if (FLEX && wid < 16 && !a.probe) {
        sh = -ilogbf(scale_a * scale_b * step_c);
        fast = sh >= 1 && sh <= 31;
        rmask = fast ? (1u << sh) - 1u : 0u;
        rhalf = fast ? 1u << (sh - 1) : 0u;
    }
    // one result: an int16 mantissa and the statistic (or what a probe wants to know); fp32 as it is
    auto finished = [&](Sum v) -> int {
        const long long x = (long long)v;
        if (a.probe) {
            const unsigned long long m = (unsigned long long)(x < 0 ? -x : x);
            pmax = m > pmax ? m : pmax;
            return 0;
        }
        const int q = fast ? rescale_i64_fast(x, sh, rmask, rhalf) : rescale_i64(x, sh), m = q < 0 ? -q : q;
        stat = m > stat ? m : stat;
        return q;
    };
    if (wid < 16) {
        ok = mbar_wait(&sums_full, 0);
        if (!ok) atomicExch(&fail_flag, 1);
        tc_fence_after();
        const unsigned lane_addr = tmem_sums + ((unsigned)(quarter * 32) << 16);
        for (int c0 = part * 4; c0 < BN; c0 += 16) {
            const int col = n0 + c0;
            if (col >= a.N) break;
            Sum v[4];
            unsigned t[3][4];
            if (FLEX) {
#pragma unroll
                for (int i = 0; i < 3; ++i) tmem_ld4(lane_addr + i * BN + c0, t[i]);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    v[j] = (Sum)(((long long)(int)t[0][j] << 16) + ((long long)(int)t[1][j] << 8) + (long long)(int)t[2][j]);
            } else {
                for (int ch = 0; ch < chains; ++ch) {
                    // (slices: chains that this one does not have count as zero)
                    if (splits == 1 || ch * kChunkKb < nkb) tmem_ld4(lane_addr + ch * BN + c0, t[0]);
                    else t[0][0] = t[0][1] = t[0][2] = t[0][3] = 0;
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float f = __uint_as_float(t[0][j]);
                        if (splits > 1) red[(ch * BN + c0 + j) * 128 + lrow] = (Sum)f;
                        else v[j] = ch ? v[j] + (Sum)f : (Sum)f;
                    }
                }
            }
            if (splits > 1) {
                if (FLEX) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) red[(c0 + j) * 128 + lrow] = v[j];
                }
                continue;
            }
            if (row >= a.M || !ok) continue;
            const int live = a.N - col;
            const long long at = a.colmajor ? (long long)col * a.ldc + row : (long long)row * a.ldc + col;
            if (FLEX) {
                int q[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) q[j] = j < live ? finished(v[j]) : 0;
                if (a.probe) continue;
                short* out = (short*)a.C + at;
                if (!a.colmajor && live >= 4 && ((uintptr_t)out & 7) == 0) {
                    *(uint2*)out = make_uint2((q[0] & 0xffff) | (q[1] << 16), (q[2] & 0xffff) | (q[3] << 16));
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j < live) out[j * (a.colmajor ? a.ldc : 1)] = (short)q[j];
                }
            } else {
                float* out = (float*)a.C + at;
                if (!a.colmajor && live >= 4 && ((uintptr_t)out & 15) == 0) {
                    *(float4*)out = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j < live) out[j * (a.colmajor ? a.ldc : 1)] = (float)v[j];
                }
            }
        }
    }
    if (splits > 1) {
        cluster_sync();
        if (wid < 16) {
            // this CTA's columns: every splits-th, dealt to the warps of a quarter, four at a time.  (A peer's values
            // take about 700 cycles: those of the four columns come together.)
            constexpr int U = BN >= 64 ? 4 : BN >= 32 ? 2 : 1;
            const int total = splits * chains, step = 4 * splits;
            for (int c = rank + part * splits; c < BN && n0 + c < a.N; c += step * U) {
                Sum v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = 0;
                constexpr int Z = 8 / U;
                for (int i0 = 0; i0 < total; i0 += Z) {
                    Sum t[Z][U];
#pragma unroll
                    for (int z = 0; z < Z; ++z) {
                        const int i = i0 + z, from = chains == 1 ? i : i / chains, ch = i - from * chains;
                        const unsigned at = i < total ? map_rank(red + (ch * BN + c) * 128 + lrow, from) : 0;
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            t[z][u] = i < total && c + u * step < BN ? ld_peer(at + u * step * 128 * (unsigned)sizeof(Sum), (Sum)0) : 0;
                    }
#pragma unroll
                    for (int z = 0; z < Z; ++z)
#pragma unroll
                        for (int u = 0; u < U; ++u) v[u] += t[z][u];
                }
                if (row >= a.M || !ok) continue;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int col = n0 + c + u * step;
                    if (c + u * step >= BN || col >= a.N) continue;
                    const long long at = a.colmajor ? (long long)col * a.ldc + row : (long long)row * a.ldc + col;
                    if (FLEX) {
                        const int q = finished(v[u]);
                        if (!a.probe) ((short*)a.C)[at] = (short)q;
                    } else {
                        ((float*)a.C)[at] = (float)v[u];
                    }
                }
            }
        }
    }
    if (FLEX && wid < 16) {
        if (a.probe) {
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long t = __shfl_xor_sync(0xffffffffu, pmax, o);
                pmax = t > pmax ? t : pmax;
            }
            if (lane == 0 && pmax) atomicMax(a.probe_out, pmax);
        } else {
            stat = __reduce_max_sync(0xffffffffu, stat);
            if (lane == 0 && stat) atomicMax(a.stats + a.slotC, stat);
        }
    }
    if (splits > 1) {                                             // (peers may still be reading)
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    if (wid == 24) {
        tc_fence_after();
        tmem_dealloc(tmem_base, p.tmem);
    }
    if (threadIdx.x == 0 && fail_flag && a.status) atomicExch(a.status, 1);
}

// ---- host ------------------------------------------------------------------------------------
struct StreamShape { int bn, splits, kb_per_split, waves; long long cost; };

inline bool str_even(const void* x, int kind, long long rs, long long ks, int size) {
    return (((uintptr_t)x | (uintptr_t)((kind == B2_OPERAND_K ? rs : ks) * size)) & 15) == 0;
}

template <int MODE>
StreamShape stream_shape(const b2_direct_args& a) {
    const int KB = MODE == MODE_FLEX16 ? 128 : 32;
    const int num_kb = (a.K + KB - 1) / KB;
    const int most = MODE == MODE_FLEX16 ? 256 : kChunkKb;        // exact int32 sums; a chain
    StreamShape best = {0, 0, 0, 0, -1};
    const long long tm = (a.M + 127) / 128;
    if (tm > 65535) return best;
    const int size = MODE == MODE_FLEX16 ? 2 : 4;
    const bool even = str_even(nullptr, a.a_kind, a.a_rs, a.a_ks, size) && str_even(nullptr, a.b_kind, a.b_rs, a.b_ks, size);
    int per_of[9] = {};                                           // k-blocks of a slice, 0: not so many slices
    for (int want = 1; want <= 8 && want <= num_kb; ++want) {
        int per = (num_kb + want - 1) / want;
        if (MODE != MODE_FLEX16 && want > 1) per = (per + most - 1) / most * most;
        if ((num_kb + per - 1) / per == want && (MODE != MODE_FLEX16 || per <= most)) per_of[want] = per;
    }
    for (int bn = 16; bn <= 128; bn *= 2) {
        if (bn > 16 && bn / 2 >= a.N) break;
        const long long tiles = tm * ((a.N + bn - 1) / bn);
        // Chains in one CTA: as many as tensor memory has sums for where the result is one narrow tile across (6673 x 23 x
        // 2680 38.1 -> 25.4 us), else one: slices of more are no faster than pairs on planes (1000 x 777 x 1500 31.4 and
        // 28.4).
        const int chains_most = MODE == MODE_FLEX16 || a.N > 32 ? 1 : (512 - str_slots(bn) * 64) / bn;
        for (int splits = 1; splits <= 8; ++splits) {
            const int per = per_of[splits], chains = MODE == MODE_FLEX16 ? 1 : (per + most - 1) / most;
            if (!per || chains > chains_most) continue;
            if (splits > 1 && chains * bn * 128 * (MODE == MODE_FLEX16 ? 8 : 4) > 200 * 1024) continue;
            // Measured on one B200 (cycles at 1.9 GHz, 1060 flex16 and 250 fp32 products, each in two shapes; the rule is
            // within 7 and 5 % of them, root mean square): lines off sixteen bytes cost their converters a shift, operands
            // by columns the loads of a column each; results by rows that are stored one by one go to as many lines
            // as there are rows; flex16 takes longer where every SM is busy.
            const long long ctas = tiles * splits, slots = kClusterCtas[splits], waves = (ctas + slots - 1) / slots;
            const int rows = a.M < 128 ? a.M : 128, live = bn < a.N ? bn : a.N, busy = ctas < 148 ? (int)ctas : 148;
            const int alone = a.colmajor || (splits == 1 && a.N % 4 == 0) ? 0 : rows * live / splits;
            const bool a_rows = a.a_kind == B2_OPERAND_ROWS, b_rows = a.b_kind == B2_OPERAND_ROWS;
            long long one, kb;
            if (MODE == MODE_FLEX16) {
                kb = 900 + 16 * bn + (even ? 0 : 470 + 6 * bn) + (a_rows ? 130 : 0);
                one = 5000 + per * kb + 84 * bn + (splits > 1 ? 1800 + 19 * bn + 5 * alone / 3 : alone) + 20 * busy - (waves > 1 ? 2300 : 0);
            } else {
                kb = 370 + 9 * bn + (even ? 0 : 155) + (a_rows ? 140 : 0) + (b_rows ? 3 * bn / 2 : 0);
                one = 6400 + per * kb + 57 * bn + (splits > 1 ? 3100 : 0) + 2 * alone / 3 - (waves > 1 ? 1300 : 0);
            }
            const long long cost = waves * one;
            if (best.cost < 0 || cost < best.cost) best = {bn, splits, per, (int)waves, cost};
        }
    }
    return best;
}

template <int MODE, int BN, int AK, int BK, bool EVEN>
int stream_launch_as(StreamParams& p, cudaStream_t st) {
    constexpr int most = str_most_stages(MODE, BN), raw = str_raw_bytes(MODE, BN, AK, BK), planes = str_slots(BN) * str_plane_bytes(BN);
    static_assert(1024 + planes + most * raw <= 232448 - 1024, "shared memory");
    const int sum = MODE == MODE_FLEX16 ? 8 : 4;
    p.stages = p.kb_per_split < most ? p.kb_per_split : most;
    int smem = planes + p.stages * raw;
    if (p.splits > 1 && p.chains * BN * 128 * sum > smem) smem = p.chains * BN * 128 * sum;      // (exchanged through it)
    smem += 1024;
    int cols = str_slots(BN) * 64 + (MODE == MODE_FLEX16 ? 3 : p.chains) * BN;
    for (p.tmem = 32; p.tmem < cols; p.tmem *= 2) {}
    static bool attr_set = false;
    if (!attr_set) {
        B2_CUDA(cudaFuncSetAttribute(stream_kernel<MODE, BN, AK, BK, EVEN>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448 - 1024));
        attr_set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.a.N + BN - 1) / BN, (p.a.M + 127) / 128, p.splits);
    cfg.blockDim = dim3(kStrThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = p.splits;
    cfg.attrs = attr;
    cfg.numAttrs = p.splits > 1 ? 2 : 1;
    B2_CUDA(cudaLaunchKernelEx(&cfg, stream_kernel<MODE, BN, AK, BK, EVEN>, p));
    return B2_OK;
}

template <int MODE, int BN, int AK, int BK>
int stream_launch_even(StreamParams& p, bool even, cudaStream_t st) {
    return even ? stream_launch_as<MODE, BN, AK, BK, true>(p, st) : stream_launch_as<MODE, BN, AK, BK, false>(p, st);
}

template <int MODE, int BN>
int stream_launch_bn(StreamParams& p, bool even, cudaStream_t st) {
    if (p.a.a_kind == B2_OPERAND_K)
        return p.a.b_kind == B2_OPERAND_K ? stream_launch_even<MODE, BN, B2_OPERAND_K, B2_OPERAND_K>(p, even, st)
                                          : stream_launch_even<MODE, BN, B2_OPERAND_K, B2_OPERAND_ROWS>(p, even, st);
    return p.a.b_kind == B2_OPERAND_K ? stream_launch_even<MODE, BN, B2_OPERAND_ROWS, B2_OPERAND_K>(p, even, st)
                                      : stream_launch_even<MODE, BN, B2_OPERAND_ROWS, B2_OPERAND_ROWS>(p, even, st);
}

template <int MODE>
int stream_launch_mode(const b2_direct_args& a, cudaStream_t st) {
    const auto& s = a.stream;
    B2_REQUIRE(s.bn > 0, "a product without a shape");
    StreamParams p;
    p.a = a;
    const int KB = MODE == MODE_FLEX16 ? 128 : 32, size = MODE == MODE_FLEX16 ? 2 : 4;
    p.num_kb = (a.K + KB - 1) / KB;
    p.kb_per_split = s.kb_per_split;
    p.splits = s.splits;
    p.chains = MODE == MODE_FLEX16 ? 1 : (s.kb_per_split + kChunkKb - 1) / kChunkKb;
    B2_REQUIRE((uintptr_t)a.A % size == 0 && (uintptr_t)a.B % size == 0, "operands must be aligned to their elements");
    const bool even = str_even(a.A, a.a_kind, a.a_rs, a.a_ks, size) && str_even(a.B, a.b_kind, a.b_rs, a.b_ks, size);
    switch (s.bn) {
        case 16: return stream_launch_bn<MODE, 16>(p, even, st);
        case 32: return stream_launch_bn<MODE, 32>(p, even, st);
        case 64: return stream_launch_bn<MODE, 64>(p, even, st);
        default: return stream_launch_bn<MODE, 128>(p, even, st);
    }
}

}  // namespace
#endif  // B2_STREAM_CUH
