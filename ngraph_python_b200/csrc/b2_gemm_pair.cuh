// The plane GEMM on pairs of SMs: C[M,N] = A * B^T from operand planes that lie K-major in scratch (see
// b2_gemm_impl.cuh for the planes and the arithmetic), one 256 x 128 tile per pair of CTAs with
// tcgen05.mma.cta_group::2.
//
// Why pairs: a 128 x 128 tile of one SM needs 64 KB of operands in shared memory per k-block, written
// once by TMA (512 cycles at 128 B/clk) and read by the instructions (768), against 1024 (flex16) and
// 768 (fp32) cycles of the tensor pipe -- shared memory, not the pipe, set its pace (1430 and 1100
// cycles a k-block measured).  In a pair each SM holds its own 128 rows of A and half of B: 48 KB
// written, 64 (72) KB read.
//   flex16: the merged operand [B_hi | B_lo'] of 256 rows is cut between the two SMs by plane:
//           A_hi x [..] -> HH | X1,  A_lo x [..] -> X2 | LL   (512 columns of tensor memory, all of it)
//   fp32:   hi*hi, hi*lo and lo*hi into one sum, in the order of the other kernels; chains of 16
//           k-blocks in two buffers, as there.
//
// Each CTA: warp 0 TMA producer (its loads complete on the leader's barrier), warp 1 tensor memory and,
// in the leader, MMA issue; warps 2-9 epilogue.  Persistent over tiles, eight tiles of rows at a time
// down the columns, so that the pairs in flight share panels in L2; the producer runs ahead into the
// next tile while the epilogue drains the last.  Where there are fewer tiles than pairs, 2 to 4 pairs
// of one cluster take slices of K and add up in distributed shared memory in slice order.  In fp32 the
// slices after the first keep up to four chains apart, each in tensor-memory columns of its own, and the
// sum takes them one by one, so that it is rounded as the kernels round it that walk all of K: a value
// near zero keeps its sign (a ReLU its mask) whatever kernel the number of rows and columns leads to.
// Slices of more chains (K > 4096, which only this kernel and the single-SM one take) add their own first.
// Against sums per slice: 1000 x 777 x 1500 32.8 -> 32.5 us, x 2048 34.5 -> 34.5, x 4096 59.7 -> 60.6,
// 768 x 512 x 4096 34.6 -> 36.0 (eight chains handed over instead of four sums; 16-byte accesses to the
// peers' memory, the sum of the first slice taken while it multiplies).
#ifndef B2_GEMM_PAIR_CUH
#define B2_GEMM_PAIR_CUH
#include "b2_direct.h"
#include "b2_gemm_impl.cuh"

namespace {

// Epilogue warps.  flex16 fills tensor memory (HH | X1 | X2 | LL), so that a tile's epilogue holds up the
// next tile's products: sixteen warps take half the time of eight.  fp32 overlaps the two, and its
// sums want the registers.
__host__ __device__ constexpr int pair_epi_warps(int mode) { return mode == MODE_FLEX16 ? 16 : 8; }
__host__ __device__ constexpr int pair_threads(int mode) { return 64 + 32 * pair_epi_warps(mode); }
constexpr int kPairStage = 48 * 1024;
constexpr int kPairStages = 4;
constexpr int kPairSmem = 1024 + kPairStages * kPairStage + 256;

// completes on a barrier of the pair's leader
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_commit_pair(unsigned long long* bar, unsigned short mask) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
        ::"r"(smem_u32(bar)), "h"(mask) : "memory");
}
__device__ __forceinline__ void arrive_remote(unsigned bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
template <int MODE>
__device__ __forceinline__ void tc_mma_pair(unsigned tmem_d, unsigned long long adesc, unsigned long long bdesc,
                                            unsigned idesc, unsigned accumulate) {
    if (MODE == MODE_FLEX16) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
    }
}
// instruction descriptor for 256 rows
__host__ __device__ constexpr unsigned idesc_pair(unsigned dfmt, unsigned afmt, unsigned bfmt, unsigned n) {
    return (dfmt << 4) | (afmt << 7) | (bfmt << 10) | ((n >> 3) << 17) | ((256u >> 4) << 24);
}
// Slices of K exchange their sums in pieces of eight columns x 128 rows.  fp32: two groups of four columns,
// rows behind one another, so that a lane's share is two 16-byte accesses and a warp's is contiguous.
__device__ __forceinline__ void put_piece(float* piece, int lrow, const float* v) {
    *(float4*)(piece + lrow * 4) = make_float4(v[0], v[1], v[2], v[3]);
    *(float4*)(piece + 512 + lrow * 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void get_piece(const float* piece, int lrow, unsigned rank, float* v) {
    const unsigned at = map_rank(piece + lrow * 4, rank);
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(at) : "memory");
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "r"(at + 2048) : "memory");
}
__device__ __forceinline__ void put_piece(long long* piece, int lrow, const long long* v) {
#pragma unroll
    for (int j = 0; j < 8; ++j) piece[j * 128 + lrow] = v[j];
}
__device__ __forceinline__ void add_piece(const float* piece, int lrow, unsigned rank, float* v) {
    float x[8];
    get_piece(piece, lrow, rank, x);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] += x[j];
}
__device__ __forceinline__ void add_piece(const long long* piece, int lrow, unsigned rank, long long* v) {
    const unsigned at = map_rank(piece + lrow, rank);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] += ld_peer(at + j * 1024, 0LL);
}

struct PairParams {
    GemmParams g;
    int tm, tn, tiles;             // 256-row and 128-column tiles
    int splits, kb_per_split;
    int apart;                     // fp32: slices after the first hand out chains, not their sum ...
    int apart_pieces, apart_inv;   // ... so many pieces of each; 32 / splits rounded up: i * inv >> 5 is i / splits, i < 16
};

constexpr int kOrderedKb = 8 * kChunkKb;   // up to here fp32 chains are added in order (K = 4096) ...
constexpr int kApartChains = 4;            // ... which leaves a slice four at most, in 128 columns each
// What slice z hands out of a chain: the pieces of eight columns that another slice finishes, one behind
// the other.  Piece round * splits + owner is finished by slice `owner`; its place in slice z's memory:
__host__ __device__ constexpr int apart_place(int round, int owner, int z, int splits) {
    return round * (splits - 1) + owner - (owner > z ? 1 : 0);
}
static_assert(kApartChains * 12 * 8 * 128 * 4 <= kPairStages * kPairStage, "12 of 16 pieces fit the ring");

// tile -> (row tile, column tile): bands of eight row tiles, down the columns
__device__ __forceinline__ void pair_tile(const PairParams& p, int t, int& m, int& n) {
    const int band = t / (8 * p.tn), in = t - band * 8 * p.tn;
    const int rows = min(8, p.tm - band * 8);
    n = in / rows;
    m = band * 8 + in - n * rows;
}

template <int MODE>
__global__ void __launch_bounds__(pair_threads(MODE), 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap mapA0, const __grid_constant__ CUtensorMap mapA1,
                 const __grid_constant__ CUtensorMap mapB0, const __grid_constant__ CUtensorMap mapB1,
                 const PairParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned long long* full_bar = (unsigned long long*)(smem + kPairStages * kPairStage);   // leader's
    unsigned long long* empty_bar = full_bar + kPairStages;
    unsigned long long* tmem_full = empty_bar + kPairStages;       // [2]
    unsigned long long* tmem_empty = tmem_full + 2;                // [2], leader's
    unsigned* tmem_holder = (unsigned*)(tmem_empty + 2);
    int* fail_flag = (int*)(tmem_holder + 1);

    const GemmParams& g = p.g;
    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    const int side = rank & 1, slice = rank >> 1;                  // of the pair, of K
    const unsigned leader = rank & ~1u;
    const unsigned short mask = (unsigned short)(3u << leader);
    constexpr int kElems = MODE == MODE_FLEX16 ? kKBytes : kKBytes / 4;
    const int kb0 = slice * p.kb_per_split;
    const int nkb = min(p.kb_per_split, g.num_kb - kb0);
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kPairStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], 2 * pair_epi_warps(MODE)); }
        *fail_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_holder)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const unsigned tmem_base = (unsigned)warp_uniform((int)*tmem_holder);

    if (warp == 0) {
        if (elect_one()) {
            int s = 0;
            unsigned parity = 1;
            bool ok = true;
            for (int t = first; t < p.tiles && ok; t += step) {
                int tm, tn;
                pair_tile(p, t, tm, tn);
                const int m0 = tm * 256 + side * 128, n0 = tn * 128;
                for (int kb = 0; kb < nkb; ++kb) {
                    if (!mbar_wait(&empty_bar[s], parity)) { atomicExch(fail_flag, 1); ok = false; break; }
                    unsigned char* st = smem + s * kPairStage;
                    const unsigned bar = map_rank(&full_bar[s], leader);
                    if (side == 0) mbar_expect_tx(&full_bar[s], 2 * kPairStage);
                    const int kx = (kb0 + kb) * kElems;
                    tma_load_2d_pair(st, &mapA0, kx, m0, bar);
                    tma_load_2d_pair(st + kPlaneBytes, &mapA1, kx, m0, bar);
                    if (MODE == MODE_FLEX16) {
                        // one plane of all 128 columns each
                        tma_load_2d_pair(st + 2 * kPlaneBytes, side ? &mapB1 : &mapB0, kx, n0, bar);
                    } else {
                        // both planes of 64 columns each
                        tma_load_2d_pair(st + 2 * kPlaneBytes, &mapB0, kx, n0 + side * 64, bar);
                        tma_load_2d_pair(st + 2 * kPlaneBytes + 64 * kKBytes, &mapB1, kx, n0 + side * 64, bar);
                    }
                    if (++s == kPairStages) { s = 0; parity ^= 1u; }
                }
            }
            // the leader's signals to this CTA's barriers must have landed before it may exit
            for (int i = 0; i < kPairStages && ok; ++i) {
                if (!mbar_wait(&empty_bar[s], parity)) { atomicExch(fail_flag, 1); ok = false; }
                if (++s == kPairStages) { s = 0; parity ^= 1u; }
            }
        }
    } else if (warp == 1) {
        if (side == 0 && elect_one()) {
            const unsigned id_s = idesc_pair(2, 1, 1, 256), id_u = idesc_pair(2, 0, 1, 256);
            const unsigned id_t = idesc_pair(1, 2, 2, 128);
            int s = 0, chunk = 0;
            unsigned parity = 0;
            bool ok = true;
            for (int t = first; t < p.tiles && ok; t += step) {
                for (int kb = 0; kb < nkb && ok; ++kb) {
                    const int kin = MODE == MODE_FLEX16 ? kb : kb % kChunkKb;
                    const bool apart = MODE != MODE_FLEX16 && p.apart && slice > 0;
                    const int b = MODE == MODE_FLEX16 || apart ? 0 : chunk & 1;
                    if (kin == 0 && !apart) {
                        // the accumulators of this chain must have been drained
                        const int use = MODE == MODE_FLEX16 ? chunk : chunk >> 1;
                        if (use > 0 && !mbar_wait(&tmem_empty[b], (use - 1) & 1)) {
                            atomicExch(fail_flag, 1); ok = false; break;
                        }
                        tc_fence_after();
                    }
                    if (!mbar_wait(&full_bar[s], parity)) { atomicExch(fail_flag, 1); ok = false; break; }
                    tc_fence_after();
                    unsigned char* st = smem + s * kPairStage;
                    const unsigned long long dA0 = make_smem_desc(st), dA1 = make_smem_desc(st + kPlaneBytes);
                    const unsigned long long dB0 = make_smem_desc(st + 2 * kPlaneBytes);
                    const unsigned long long dB1 = make_smem_desc(st + 2 * kPlaneBytes + 64 * kKBytes);
                    const unsigned acc0 = tmem_base + (apart ? (kb / kChunkKb) * 128 : b * 256);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const unsigned long long adv = (unsigned long long)(2 * k);
                        const unsigned acc = (kin > 0 || k > 0) ? 1u : 0u;
                        if (MODE == MODE_FLEX16) {
                            tc_mma_pair<MODE>(tmem_base, dA0 + adv, dB0 + adv, id_s, acc);          // HH | X1
                            tc_mma_pair<MODE>(tmem_base + 256, dA1 + adv, dB0 + adv, id_u, acc);    // X2 | LL
                        } else {
                            tc_mma_pair<MODE>(acc0, dA0 + adv, dB0 + adv, id_t, acc);               // hi*hi
                            // (into one sum, in the single-SM kernel's order: the same rounding)
                            tc_mma_pair<MODE>(acc0, dA0 + adv, dB1 + adv, id_t, 1u);                // hi*lo
                            tc_mma_pair<MODE>(acc0, dA1 + adv, dB0 + adv, id_t, 1u);                // lo*hi
                        }
                    }
                    tc_commit_pair(&empty_bar[s], mask);
                    if (++s == kPairStages) { s = 0; parity ^= 1u; }
                    if (kb == nkb - 1 || (MODE != MODE_FLEX16 && !apart && kin == kChunkKb - 1)) {
                        tc_commit_pair(&tmem_full[b], mask);
                        ++chunk;
                    }
                }
            }
        }
    } else {
        // epilogue: lane quarter = warp % 4, a share of the columns each
        typedef typename std::conditional<MODE == MODE_FLEX16, long long, float>::type Sum;
        Sum* red = (Sum*)smem;                                    // 16 pieces (of every chain, apart), slices only
        constexpr int kGroups = pair_epi_warps(MODE) / 4, kCols = 128 / kGroups;
        const int quarter = warp & 3, c_lo = ((warp - 2) >> 2) * kCols;
        const int lrow = quarter * 32 + lane;
        const unsigned lane_addr = tmem_base + ((unsigned)(quarter * 32) << 16);
        const unsigned empty0 = map_rank(&tmem_empty[0], leader), empty1 = map_rank(&tmem_empty[1], leader);
        bool ok = true;
        int stat = 0, sh = 0, chunk = 0;
        unsigned long long pmax = 0;
        if (MODE == MODE_FLEX16)
            sh = -ilogbf(g.table[g.slotA].scale * g.table[g.slotB].scale * (g.probe ? 1.0f : g.table[g.slotC].inv_scale));
        const bool fast = sh >= 1 && sh <= 31;
        const unsigned rmask = fast ? (1u << sh) - 1u : 0u, rhalf = fast ? 1u << (sh - 1) : 0u;
        // eight finished sums of one row
        auto finish = [&](int row, int col, long long fix, const Sum* v) {
            if (row >= g.M || col >= g.N) return;
            const int live = g.N - col;
            if (MODE == MODE_FLEX16) {
                int q[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const long long x = (long long)v[j] + fix;
                    if (g.probe) {
                        const unsigned long long m = (unsigned long long)(x < 0 ? -x : x);
                        if (j < live) pmax = m > pmax ? m : pmax;
                    } else {
                        q[j] = fast ? rescale_i64_fast(x, sh, rmask, rhalf) : rescale_i64(x, sh);
                        const int m = q[j] < 0 ? -q[j] : q[j];
                        if (j < live) stat = m > stat ? m : stat;
                    }
                }
                if (g.probe) return;
                short* out = (short*)g.C + (long long)row * g.ldc + col;
                if (live >= 8 && ((uintptr_t)out & 15) == 0) {
                    uint4 w;
                    w.x = (q[0] & 0xffff) | (q[1] << 16); w.y = (q[2] & 0xffff) | (q[3] << 16);
                    w.z = (q[4] & 0xffff) | (q[5] << 16); w.w = (q[6] & 0xffff) | (q[7] << 16);
                    *(uint4*)out = w;
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (j < live) out[j] = (short)q[j];
                }
            } else {
                float* out = (float*)g.C + (long long)row * g.ldc + col;
                if (live >= 8 && ((uintptr_t)out & 15) == 0) {
                    *(float4*)out = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
                    *(float4*)(out + 4) = make_float4((float)v[4], (float)v[5], (float)v[6], (float)v[7]);
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (j < live) out[j] = (float)v[j];
                }
            }
        };
        for (int t = first; t < p.tiles; t += step) {
            int tm, tn;
            pair_tile(p, t, tm, tn);
            const int row = tm * 256 + side * 128 + lrow, n0 = tn * 128;
            const long long fix = MODE == MODE_FLEX16 && row < g.M ? 128LL * (long long)g.rowsum[row] : 0LL;
            if (MODE == MODE_FLEX16) {
                if (ok && !mbar_wait(&tmem_full[0], chunk & 1)) { atomicExch(fail_flag, 1); ok = false; }
                ++chunk;
                tc_fence_after();
                for (int c0 = c_lo; c0 < c_lo + kCols; c0 += 8) {
                    unsigned hh[8], x1[8], x2[8], ll[8];
                    tmem_ld8(lane_addr + c0, hh);
                    tmem_ld8(lane_addr + 128 + c0, x1);
                    tmem_ld8(lane_addr + 256 + c0, x2);
                    tmem_ld8(lane_addr + 384 + c0, ll);
                    tmem_ld_wait();
                    Sum v[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        v[j] = (Sum)(((long long)(int)hh[j] << 16) +
                                     (((long long)(int)x1[j] + (long long)(int)x2[j]) << 8) + (long long)(int)ll[j]);
                    if (p.splits > 1) {
                        put_piece(red + c0 * 128, lrow, v);
                    } else if (ok) {
                        finish(row, n0 + c0, fix, v);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) arrive_remote(empty0);
            } else if (p.apart && slice > 0) {
                // (one tile per cluster)  all products are done: the ring is free
                if (ok && !mbar_wait(&tmem_full[0], 0)) { atomicExch(fail_flag, 1); ok = false; }
                tc_fence_after();
                const int pieces = p.apart_pieces;
                for (int ch = 0; ch * kChunkKb < nkb; ++ch)
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        const int i0 = (c_lo >> 3) + 4 * half;
                        unsigned v[32];
                        tmem_ld16(lane_addr + ch * 128 + i0 * 8, v);
                        tmem_ld16(lane_addr + ch * 128 + i0 * 8 + 16, v + 16);
                        tmem_ld_wait();
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int round = (i0 + u) * p.apart_inv >> 5, owner = i0 + u - round * p.splits;
                            if (owner == slice) continue;
                            Sum x[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) x[j] = (Sum)__uint_as_float(v[8 * u + j]);
                            put_piece(red + (ch * pieces + apart_place(round, owner, slice, p.splits)) * 8 * 128, lrow, x);
                        }
                    }
            } else {
                Sum sum[64];
#pragma unroll
                for (int j = 0; j < 64; ++j) sum[j] = 0;
                const int chunks = (nkb + kChunkKb - 1) / kChunkKb;
                for (int i = 0; i < chunks; ++i, ++chunk) {
                    const int b = chunk & 1;
                    if (ok && !mbar_wait(&tmem_full[b], (chunk >> 1) & 1)) { atomicExch(fail_flag, 1); ok = false; }
                    tc_fence_after();
#pragma unroll
                    for (int c0 = 0; c0 < 64; c0 += 16) {
                        unsigned v[16];
                        tmem_ld16(lane_addr + b * 256 + c_lo + c0, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) sum[c0 + j] += (Sum)__uint_as_float(v[j]);
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) arrive_remote(b ? empty1 : empty0);
                }
#pragma unroll
                for (int c0 = 0; c0 < 64; c0 += 8) {
                    if (p.splits > 1) {
                        put_piece(red + (c_lo + c0) * 128, lrow, sum + c0);
                    } else if (ok) {
                        finish(row, n0 + c_lo + c0, 0, sum + c0);
                    }
                }
            }
        }
        if (p.splits > 1) {
            // (one tile per cluster)  every slice adds a share of the column pieces
            cluster_sync();
            int tm, tn;
            pair_tile(p, first, tm, tn);
            const int row = tm * 256 + side * 128 + lrow, n0 = tn * 128;
            const long long fix = MODE == MODE_FLEX16 && row < g.M ? 128LL * (long long)g.rowsum[row] : 0LL;
            // piece round * splits + slice of eight columns
            for (int round = (warp - 2) >> 2; round * p.splits + slice < 16; round += kGroups) {
                const int c0 = (round * p.splits + slice) * 8;
                Sum v[8];
                bool whole = true;                                // every slice hands out its sum
                if constexpr (MODE != MODE_FLEX16) if (p.apart) {
                    whole = false;
                    get_piece(red + c0 * 128, lrow, side, v);
                    // the chains of the other slices, four at a time in flight
                    const int per = p.kb_per_split / kChunkKb;
                    const int chains = (g.num_kb - p.kb_per_split + kChunkKb - 1) / kChunkKb;
                    int z = 1, ch = 0;
                    for (int q = 0; q < chains; q += 4) {
                        Sum x[4][8];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (q + u >= chains) break;
                            if (z == slice) {
                                unsigned y[8];
                                tmem_ld8(lane_addr + ch * 128 + c0, y);
                                tmem_ld_wait();
#pragma unroll
                                for (int j = 0; j < 8; ++j) x[u][j] = (Sum)__uint_as_float(y[j]);
                            } else {
                                const int at = ch * p.apart_pieces + apart_place(round, slice, z, p.splits);
                                get_piece(red + at * 8 * 128, lrow, 2 * z + side, x[u]);
                            }
                            if (++ch == per) { ch = 0; ++z; }
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (q + u >= chains) break;
#pragma unroll
                            for (int j = 0; j < 8; ++j) v[j] += x[u][j];
                        }
                    }
                }
                if (whole) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = 0;
                    for (int z = 0; z < p.splits; ++z) add_piece(red + c0 * 128, lrow, 2 * z + side, v);
                }
                if (ok) finish(row, n0 + c0, fix, v);
            }
        }
        if (MODE == MODE_FLEX16) {
            if (g.probe) {
                for (int o = 16; o > 0; o >>= 1) {
                    const unsigned long long x = __shfl_xor_sync(0xffffffffu, pmax, o);
                    pmax = x > pmax ? x : pmax;
                }
                if (lane == 0 && pmax) atomicMax(g.probe_out, pmax);
            } else {
                for (int o = 16; o > 0; o >>= 1) {
                    const int x = __shfl_xor_sync(0xffffffffu, stat, o);
                    stat = x > stat ? x : stat;
                }
                if (lane == 0 && stat) atomicMax(g.stats + g.slotC, stat);
            }
        }
    }
    __syncwarp();
    if (warp < 2 && p.splits > 1) cluster_sync();             // (the epilogue's exchange)
    tc_fence_before();
    cluster_sync();               // nothing of the pair is still to be read or signalled
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
    if (threadIdx.x == 0 && *fail_flag && g.status) atomicExch(g.status, 1);
}

// Clusters of `splits` pairs that the machine holds at once: 74, 33, 22, 15 (a cluster stays within a GPC)
inline int pair_clusters(int splits) { return kClusterCtas[2 * splits] / (2 * splits); }
inline long long pair_waves(int tiles, int splits) { return (tiles + pair_clusters(splits) - 1) / pair_clusters(splits); }
// k-blocks of a slice; fp32 slices are whole chains
inline int pair_slice(int mode, int num_kb, int splits) {
    const int per = (num_kb + splits - 1) / splits;
    return mode == MODE_FLEX16 || splits == 1 ? per : (per + kChunkKb - 1) / kChunkKb * kChunkKb;
}
// As many slices as leave every tile's cluster a place in the first wave: with one more a few clusters
// would wait for all the others.  35 tiles, 1280 x 896 x 2048: 56.3 us in two slices, 48.2 in one (flex16
// 39.7, 29.0); 16 tiles, 1024 x 512 x 4096: 57.2 us in four, 45.6 in three (flex16 43.8, 32.4).
inline int pair_splits(int mode, int tiles, int num_kb) {
    for (int s = 4; s > 1; --s) {
        if (tiles > pair_clusters(s) || (mode == MODE_FLEX16 ? num_kb < 4 * s : num_kb <= kChunkKb * (s / 2))) continue;
        const int per = pair_slice(mode, num_kb, s);
        return (num_kb + per - 1) / per;
    }
    return 1;
}

// The planes are in scratch, A's rows padded to 256 and B's to 128.
template <int MODE>
int launch_pair(unsigned char* base, const Shapes& s, GemmParams g, cudaStream_t st) {
    int rc = get_encode();
    if (rc) return rc;
    const size_t a_plane = (size_t)s.Mp * s.Kp * s.esize, b_plane = (size_t)s.Np * s.Kp * s.esize;
    CUtensorMap mA0, mA1, mB0, mB1;
    const int b_rows = MODE == MODE_FLEX16 ? 128 : 64;
    if ((rc = make_map(&mA0, base, s.Mp, s.Kp, s.esize, 128))) return rc;
    if ((rc = make_map(&mA1, base + a_plane, s.Mp, s.Kp, s.esize, 128))) return rc;
    if ((rc = make_map(&mB0, base + 2 * a_plane, s.Np, s.Kp, s.esize, b_rows))) return rc;
    if ((rc = make_map(&mB1, base + 2 * a_plane + b_plane, s.Np, s.Kp, s.esize, b_rows))) return rc;
    PairParams p;
    p.g = g;
    p.g.num_kb = s.Kp / (kKBytes / s.esize);
    p.tm = (g.M + 255) / 256; p.tn = (g.N + 127) / 128; p.tiles = p.tm * p.tn;
    p.splits = pair_splits(MODE, p.tiles, p.g.num_kb);
    p.kb_per_split = pair_slice(MODE, p.g.num_kb, p.splits);
    p.apart_pieces = 16 - 16 / p.splits;
    p.apart_inv = (32 + p.splits - 1) / p.splits;
    p.apart = MODE != MODE_FLEX16 && p.splits > 1 && p.g.num_kb <= kOrderedKb;
    static bool attr_set = false;
    if (!attr_set) {
        B2_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem));
        attr_set = true;
    }
    cudaLaunchConfig_t cfg = {};
    const int pairs = p.splits > 1 || p.tiles < 74 ? p.tiles : 74;
    cfg.gridDim = dim3(2 * pairs, 1, p.splits);
    cfg.blockDim = dim3(pair_threads(MODE));
    cfg.dynamicSmemBytes = kPairSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = p.splits;
    cfg.attrs = attr; cfg.numAttrs = 2;
    B2_CUDA(cudaLaunchKernelEx(&cfg, gemm_pair_kernel<MODE>, mA0, mA1, mB0, mB1, p));
    return B2_OK;
}

}  // namespace
#endif  // B2_GEMM_PAIR_CUH
