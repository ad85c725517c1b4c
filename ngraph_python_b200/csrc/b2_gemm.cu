// C-ABI entry points of the dense GEMM (the kernels and their launch helpers are in
// b2_gemm_impl.cuh, which the convolution entry points share).
#define B2_GEMM_OWNS_TILE_KERNEL
#include "b2_direct.h"
#include "b2_gemm_impl.cuh"
#include "b2_gemm_pair.cuh"

int b2_gemm_launch_on_planes(int mode, unsigned char* base, const void* shapes, const void* params,
                             cudaStream_t st, int splits, void* workspace) {
    const Shapes& s = *static_cast<const Shapes*>(shapes);
    const GemmParams& p = *static_cast<const GemmParams*>(params);
    return mode == MODE_FLEX16
        ? launch_on_planes<MODE_FLEX16>(base, s, p, st, splits, workspace)
        : launch_on_planes<MODE_F32X3>(base, s, p, st, splits, workspace);
}

namespace {
// Pairs of SMs take every product of more than one row tile and more than 64 columns (and sums that
// fit one slice); the single-SM tile kernel keeps the narrow ones.
inline bool goes_in_pairs(const Shapes& s, int M, int splits) {
    return s.bn == 128 && M > kBlockM && splits == 1;
}

// Cycles of the plane path: the pre-pass launch, its traffic, and the tile kernel at the cycles measured for a
// k-block.  (2500 cycles less, for the launch that two operands share, sends products the wrong way: flex16
// 2165 x 116 x 1878 22 us direct, 34 on planes, 1121 x 705 x 489 23 and 29; fp32 942 x 2897 x 54 24 and 27.)
inline long long plane_cost(int mode, const Shapes& s, int M, int N, int K) {
    const long long prepass = ((long long)M + N) * K * (mode == MODE_FLEX16 ? 4 : 12) / 2600;
    const long long num_kb = s.Kp / (kKBytes / s.esize);
    if (goes_in_pairs(s, M, pick_splits(mode, s, false))) {
        const int tiles = ((M + 255) / 256) * ((N + 127) / 128), z = pair_splits(mode, tiles, (int)num_kb);
        const long long kb = mode == MODE_FLEX16 ? 1100 : 900;
        return (mode == MODE_FLEX16 ? 20000 : 14000) + prepass +
               pair_waves(tiles, z) * (5000 + pair_slice(mode, (int)num_kb, z) * kb) + (z > 1 ? 2500 : 0);
    }
    const long long kb = (mode == MODE_FLEX16 ? 1430LL : 1100LL) * (128 + s.bn) / 256;
    const long long tiles = (long long)(s.Mp / kBlockM) * (s.Np / s.bn);
    return (mode == MODE_FLEX16 ? 20000 : 13000) + prepass + (tiles + 147) / 148 * (3500 + num_kb * kb);
}

// The same for flex16 products that the kernel of b2_stream.cuh may take instead, with what the rule above leaves out:
// results that are stored one by one, operands that do not start their lines on sixteen bytes (7053 x 271 x 336 takes 50
// us on planes, 5282 x 5707 x 137 318).
inline long long plane_cost_measured(const b2_direct_args& d, long long plane) {
    const long long results = (long long)d.M * d.N;
    return plane + 3000 + results * (d.N % 8 == 0 ? 0 : d.N % 4 == 0 ? 9 : 16) / 1000 +
           (b2_product_even(d) ? 0 : ((long long)d.M + d.N) * d.K * 2 / 1000);
}

// A product in one launch: the kernel that takes least for it, and C or its transpose -- so that a product with few rows
// does not pad them to a whole tile.  `out` gets its arguments; whether that takes less than the planes.
//
// Both kernels and the planes measured side by side on one B200, 1900 products of 1 to 8192 rows, columns and K in all
// three layouts:
//   fp32, the cheaper of b2_stream.cuh's cost and b2_direct.cuh's, which is short by 1.4 where both operands are
//     contiguous along their rows and by 1.05 elsewhere (512 x 128 x 512 8.6 us against 10.7, 1784 x 508 x 952
//     transposed 31.6 and 23.9, 1489 x 605 x 176 13.3 and 12.7), of 129 to 1024 columns or narrow results, and where no
//     line has to be shifted out of words that its neighbour shares (99 x 1347 x 2389 19.3 and 17.0).
//   flex16, b2_stream.cuh's, 1.36 times as fast (geometric mean), but
//     for one k-block and many results, where the other's two CTAs an SM hide the epilogue (2929 x 567 x 122 22.5 and 16.2);
//     for one k-block and few results whose operands lie along K off sixteen bytes (7 x 128 x 31 4.9 and 4.1);
//     for narrow results with many k-blocks to a CTA, both operands along K and on sixteen bytes (78 x 3096 x 3360 21.7
//     and 17.9, 4396 x 44 x 5248 21.0 and 18.5).
inline bool gemm_goes_direct(int mode, const void* A, long long a_rs, long long a_cs, const void* B,
                             long long b_ks, long long b_ns, int M, int N, int K, b2_direct_args* out, bool may_stream = true) {
    b2_direct_args d = {};
    d.flex = mode == MODE_FLEX16;
    d.A = A; d.a_rs = a_rs; d.a_ks = a_cs; d.a_kind = a_cs == 1 ? B2_OPERAND_K : B2_OPERAND_ROWS;
    d.B = B; d.b_rs = b_ns; d.b_ks = b_ks; d.b_kind = b_ks == 1 ? B2_OPERAND_K : B2_OPERAND_ROWS;
    d.M = M; d.N = N; d.K = K;
    b2_direct_args t = d;
    t.A = d.B; t.a_rs = d.b_rs; t.a_ks = d.b_ks; t.a_kind = d.b_kind;
    t.B = d.A; t.b_rs = d.a_rs; t.b_ks = d.a_ks; t.b_kind = d.a_kind;
    t.M = N; t.N = M; t.colmajor = 1;
    const bool by_rows = d.a_kind == B2_OPERAND_ROWS && d.b_kind == B2_OPERAND_ROWS;
    const bool along_k = d.a_kind == B2_OPERAND_K && d.b_kind == B2_OPERAND_K, even = b2_product_even(d);
    const long long plane = plane_cost(mode, shapes_for(mode, M, N, K), M, N, K), results = (long long)M * N;
    auto cheaper = [&](long long cd, long long ct) {
        const bool swap = ct >= 0 && (cd < 0 || ct < cd);
        *out = swap ? t : d;
        return swap ? ct : cd;
    };
    long long stream = -1;
    if (may_stream && mode == MODE_FLEX16) {
        const bool few = along_k && !even && M <= 64 && results < 4096;
        if (K > 128 || (!few && results < (by_rows || along_k ? 900000 : 400000))) {
            // (near each other C itself is the faster: 178 x 2 x 46 transposed 4.2 and 4.7 us)
            const long long ct = b2_stream_cost(t);
            stream = cheaper(b2_stream_cost(d), ct < 0 ? ct : ct + 1000);
            out->streams = 1;
            if (along_k && even && K > 13 * 128 && stream >= 0 && (M <= 192 || N <= 192)) {
                if (out->stream.kb_per_split >= 14) {
                    const b2_direct_args streamed = *out;
                    const long long direct = cheaper(b2_direct_cost(d), b2_direct_cost(t));
                    if (direct < 0 || direct >= stream + stream * 2 / 9) *out = streamed;
                }
            }
            // (many k-blocks in few slices: flex16 500 x 500 x 6000, the second operand along K, 19.7 us on planes, 21.6
            // in one launch)
            if (K > 4096 && M > 256 && N > 256) return stream >= 0 && stream + stream / 8 < plane;
            return stream >= 0 && stream < (K > 128 ? plane_cost_measured(d, plane) : plane);
        }
    } else if (may_stream && K > 128 && (K <= 1024 || M <= 32 || N <= 32) && (by_rows || even)) {
        stream = cheaper(b2_stream_cost(d), b2_stream_cost(t));
    }
    const b2_direct_args streamed = *out;
    long long best = cheaper(b2_direct_cost(d), b2_direct_cost(t));
    if (stream >= 0 && stream < plane && (best < 0 || stream <= best + (by_rows ? best * 2 / 5 : best / 20))) {
        *out = streamed;
        out->streams = 1;
        return true;
    }
    // Both operands contiguous along their rows take longer than the direct kernel's own choice of a shape has to
    // know: fp32 638 x 937 x 631 26 us against 20 on planes, 383 x 3300 x 1440 47 and 39 (two k-blocks or less
    // don't: 1869 x 1337 x 46 20 and 26); flex16 an odd number of values apart, loaded one by one, 249 x 1831 x
    // 3065 75 and 41, 745 x 913 x 1135 65 and 31.  (With one of the two along K: 236 x 339 x 3450 26 and 33.)
    if (by_rows) {
        if (mode == MODE_F32X3) best += K > 64 ? best / 6 : 0;
        else if (K > 128 && out->a_ks % 2 != 0) best += best / 2;
    }
    return best >= 0 && best < plane;
}

template <typename T, int MODE>
int run_gemm(const T* A, long long a_rs, long long a_cs, const T* B, long long b_ks, long long b_ns,
             void* C, long long ldc, int M, int N, int K, const b2_flex_scale* table, int slotA,
             int slotB, int slotC, int* stats, void* scratch, size_t scratch_bytes,
             unsigned long long* probe_out, int* status, int probe, cudaStream_t st) {
    B2_REQUIRE(A && B && C && M > 0 && N > 0 && K > 0, "bad GEMM argument");
    B2_REQUIRE(a_rs == 1 || a_cs == 1, "A must be contiguous along M or K");
    B2_REQUIRE(b_ks == 1 || b_ns == 1, "B must be contiguous along K or N");
    const Shapes s = shapes_for(MODE, M, N, K);
    const size_t need = gemm_scratch_need(MODE, s);
    const bool room = scratch && scratch_bytes >= need && ((uintptr_t)scratch & 1023) == 0;
    b2_direct_args d;
    // (what needs scratch does not change with the kernels' measurements: without it one launch takes what
    // b2_direct.cuh's kernel would be chosen for)
    if (!room)
        B2_REQUIRE(gemm_goes_direct(MODE, A, a_rs, a_cs, B, b_ks, b_ns, M, N, K, &d, false),
                   "GEMM needs %zu bytes of 1024-byte aligned scratch, got %zu", need, scratch_bytes);
    if (gemm_goes_direct(MODE, A, a_rs, a_cs, B, b_ks, b_ns, M, N, K, &d) || !room) {
        d.C = C; d.ldc = ldc; d.table = table; d.slotC = slotC;
        d.slotA = d.colmajor ? slotB : slotA; d.slotB = d.colmajor ? slotA : slotB;
        d.stats = stats; d.probe_out = probe_out; d.status = status; d.probe = probe;
        return d.streams ? b2_stream_launch(d, st) : b2_direct_launch(d, st);
    }
    const int splits = pick_splits(MODE, s, false);     // > 1 only for flex16 with K > 32768
    unsigned char* base = (unsigned char*)scratch;
    const size_t a_plane = (size_t)s.Mp * s.Kp * s.esize, b_plane = (size_t)s.Np * s.Kp * s.esize;
    void* A0 = base; void* A1 = base + a_plane;
    void* B0 = base + 2 * a_plane; void* B1 = base + 2 * a_plane + b_plane;
    int* rowsum = nullptr;
    unsigned lo_xor = 0;
    if (MODE == MODE_FLEX16) {
        rowsum = (int*)(base + s.rowsum_off);
        lo_xor = 0x80;
    }
    const SplitJob ja = split_job<T, MODE>(A, a_rs, a_cs, M, K, s.Mp, s.Kp, A0, A1, 0, rowsum);
    if (rowsum && ja.way != kSplitRowSums) B2_CUDA(cudaMemsetAsync(rowsum, 0, (size_t)s.Mp * sizeof(int), st));
    // op(B)^T: rows = N, element (n, k) = B[k * b_ks + n * b_ns]
    const SplitJob jb = split_job<T, MODE>(B, b_ns, b_ks, N, K, s.Np, s.Kp, B0, B1, lo_xor, nullptr);
    const int rc = split_operands<T, MODE>(ja, jb, st);
    if (rc) return rc;
    GemmParams p;
    p.M = M; p.N = N; p.num_kb = 0;
    p.ldc = ldc; p.C = C; p.table = table; p.slotA = slotA; p.slotB = slotB; p.slotC = slotC;
    p.stats = stats; p.probe_out = probe_out; p.status = status; p.probe = probe;
    p.c_colmajor = 0;
    p.rowsum = rowsum;
    if (goes_in_pairs(s, M, splits)) return launch_pair<MODE>(base, s, p, st);
    return launch_on_planes<MODE>(base, s, p, st, splits, base + align1k(s.bytes));
}

}  // namespace

extern "C" int b2_gemm_scratch_bytes(int32_t flex, int32_t M, int32_t N, int32_t K, size_t* bytes) {
    B2_REQUIRE(bytes && M > 0 && N > 0 && K > 0, "bad argument");
    const int mode = flex ? MODE_FLEX16 : MODE_F32X3;
    *bytes = gemm_scratch_need(mode, shapes_for(mode, M, N, K));
    return B2_OK;
}

extern "C" int b2_gemm_route(int32_t flex, int64_t a_rs, int64_t a_cs, int64_t b_ks, int64_t b_ns, int32_t M, int32_t N,
                             int32_t K, b2_gemm_plan_info* plan, int32_t* launches) {
    B2_REQUIRE(plan && launches && M > 0 && N > 0 && K > 0, "bad argument");
    B2_REQUIRE((a_rs == 1 || a_cs == 1) && (b_ks == 1 || b_ns == 1), "operands are contiguous along one of their sides");
    const int mode = flex ? MODE_FLEX16 : MODE_F32X3;
    b2_direct_args d;
    if (gemm_goes_direct(mode, nullptr, a_rs, a_cs, nullptr, b_ks, b_ns, M, N, K, &d)) {
        *launches = 1;
        if (d.streams) {
            *plan = {B2_GEMM_STREAM, d.stream.bn, d.stream.splits, d.stream.waves};
        } else {
            b2_direct_plan(d, plan);
        }
        return B2_OK;
    }
    const Shapes s = shapes_for(mode, M, N, K);
    const int splits = pick_splits(mode, s, false);
    *launches = splits > 1 ? 3 : 2;
    if (goes_in_pairs(s, M, splits)) {
        const int tiles = ((M + 255) / 256) * ((N + 127) / 128), z = pair_splits(mode, tiles, (int)(s.Kp / (kKBytes / s.esize)));
        *plan = {B2_GEMM_PAIRS, 128, z, (int)pair_waves(tiles, z)};
    } else {
        *plan = {B2_GEMM_TILES, s.bn, splits, (int)(((long long)(s.Mp / kBlockM) * (s.Np / s.bn) * splits + 147) / 148)};
    }
    return B2_OK;
}

extern "C" int b2_gemm_launches(int32_t flex, int64_t a_k_stride, int64_t b_k_stride, int32_t M,
                                int32_t N, int32_t K, int32_t* launches) {
    b2_gemm_plan_info plan;
    return b2_gemm_route(flex, a_k_stride == 1 ? K : 1, a_k_stride, b_k_stride, b_k_stride == 1 ? K : 1, M, N, K, &plan, launches);
}

extern "C" int b2_gemm_plan(int32_t flex, int64_t a_k_stride, int64_t b_k_stride, int32_t M, int32_t N,
                            int32_t K, b2_gemm_plan_info* plan) {
    int32_t launches;
    const int rc = b2_gemm_route(flex, a_k_stride == 1 ? K : 1, a_k_stride, b_k_stride, b_k_stride == 1 ? K : 1, M, N, K, plan, &launches);
    if (rc == B2_OK && plan->kernel == B2_GEMM_STREAM) plan->kernel = B2_GEMM_DIRECT;
    return rc;
}

extern "C" int b2_gemm_f32(const float* A, int64_t a_row_stride, int64_t a_k_stride, const float* B,
                           int64_t b_k_stride, int64_t b_col_stride, float* C, int64_t ldc,
                           int32_t M, int32_t N, int32_t K, void* scratch, size_t scratch_bytes,
                           int32_t* status, void* stream) {
    return run_gemm<float, MODE_F32X3>(A, a_row_stride, a_k_stride, B, b_k_stride, b_col_stride, C,
                                       ldc, M, N, K, nullptr, 0, 0, 0, nullptr, scratch,
                                       scratch_bytes, nullptr, status, 0, (cudaStream_t)stream);
}

extern "C" int b2_gemm_flex16(const int16_t* A, int64_t a_row_stride, int64_t a_k_stride,
                              const int16_t* B, int64_t b_k_stride, int64_t b_col_stride,
                              int16_t* C, int64_t ldc, int32_t M, int32_t N, int32_t K,
                              const b2_flex_scale* table, int32_t slotA, int32_t slotB,
                              int32_t slotC, int32_t* stats, void* scratch, size_t scratch_bytes,
                              uint64_t* probe_out, int32_t* status, int32_t probe, void* stream) {
    B2_REQUIRE(table && slotA >= 0 && slotB >= 0 && slotC >= 0, "flex GEMM needs the scale table");
    B2_REQUIRE(probe ? probe_out != nullptr : stats != nullptr, "missing statistics destination");
    return run_gemm<short, MODE_FLEX16>(A, a_row_stride, a_k_stride, B, b_k_stride, b_col_stride, C,
                                        ldc, M, N, K, table, slotA, slotB, slotC, stats, scratch,
                                        scratch_bytes, (unsigned long long*)probe_out, status,
                                        probe ? 1 : 0, (cudaStream_t)stream);
}

// ---- self-test of the bounded-wait path ----------------------------------------------------------
// Every device-side wait of the tile kernels (on an mbarrier that a TMA copy, an MMA commit or
// another warp completes) gives up after a fixed number of polls, sets the caller's status word
// and lets the kernel finish normally -- tensor memory freed, nothing left spinning.  This kernel
// runs exactly that path on purpose and harmlessly: it waits, with the kernels' own wait routine,
// on a barrier that nothing will ever complete, for `poll_limit` polls, then reports and cleans up
// as the tile kernels do.  No fault, no trap, no endless loop: the context stays usable.
namespace {
__global__ void __launch_bounds__(64)
bounded_wait_selftest_kernel(int poll_limit, int* status, int* waited_out) {
    __shared__ unsigned long long bar;
    __shared__ unsigned holder;
    __shared__ int failed;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);                    // one arrival expected; nobody arrives
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(&holder, 32);    // held across the wait, like the tile kernels
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 32 && !mbar_wait_limit(&bar, 0, poll_limit)) atomicExch(&failed, 1);
    __syncthreads();
    if (threadIdx.x == 0 && failed) {
        if (status) atomicExch(status, 1);
        if (waited_out) *waited_out = poll_limit;
    }
    if (warp == 0) tmem_dealloc(holder, 32);
}
}  // namespace

extern "C" int b2_selftest_bounded_wait(int32_t poll_limit, int32_t* status, int32_t* polls_waited,
                                        void* stream) {
    B2_REQUIRE(poll_limit > 0 && poll_limit <= (1 << 16), "poll limit must be in 1..65536");
    B2_REQUIRE(status, "null status word");
    bounded_wait_selftest_kernel<<<1, 64, 0, (cudaStream_t)stream>>>(poll_limit, status, polls_waited);
    B2_CUDA(cudaGetLastError());
    return B2_OK;
}
