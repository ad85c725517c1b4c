// Tensor-core product with the operands converted on the way in: C[M,N] = A[M,K] * B[N,K]^T in one
// launch, for problems where the pre-pass of the plane kernel (b2_gemm_impl.cuh) and its launches
// cost as much as the product, and for convolutions that would otherwise be unrolled in memory.  (Matrix products
// of more than a few k-blocks: b2_stream.cuh.)
//
// One CTA per 128 x BN tile (times a slice of K), 288 or 544 threads:
//   one or two groups of eight warps: producers -- load a k-block of both operands from wherever it
//              lies (K contiguous, rows contiguous, or rows gathered from a C,H,W,N tensor through a
//              table of column offsets), split it into its two planes and store them K-major, 128-byte
//              swizzled, into a ring of stages, the groups by turns; the first group afterwards the epilogue;
//   one warp:  tensor memory, tcgen05.mma issue;
//   one more where B lies ready as the stages hold it: its copies.
// A k-block is 128 bytes of plane: 32 fp32 or 128 int16 values.
//   fp32:   3xTF32, in chains of at most 16 k-blocks (the tensor core's fp32 sum truncates); longer K
//           is cut into slices.  Matrix products add hi*hi, hi*lo and lo*hi into one sum (see ONE_CHAIN).
//           Convolutions keep two: B's planes lie behind one another and make one operand of 2*BN rows,
//           A_hi x [B_hi | B_lo] -> [hh | x], A_lo x B_hi -> x.  The sum in tensor memory loses
//           bits with every k-block, so the k-blocks go by turns to two pairs, or four where tensor memory has room,
//           which are added to nearest at the end: against 64 bits, the shapes of the 22-layer networks at
//           batch 1 to 1000, most errors are half of what they are with one pair (16 channels at 32x32,
//           batch 100, 5.0e-7 -> 2.9e-7 of the result's root mean square), for one percent of the time.  No shape may
//           put more k-blocks into one sum than with one pair (b2_direct_args::longest): of 336 random layers and
//           passes the errors against 64 bits are 0.70 of those with one pair (geometric mean), none larger by more than 3 %
//           (of K of 75); without that bound 54 of 8010 shapes had longer sums and up to 1.4 times the error.
//   flex16: four exact int8 products, HH | X | LL as in b2_gemm_impl.cuh.
// Slices of K: the CTAs of a cluster (up to 8) take one each; partial sums meet in distributed shared
// memory, every CTA adds a share of the columns in slice order (deterministic, fp32 adds rounded to
// nearest, flex16 exact in int64) and finishes them.
//
// What bounds it: at the sizes it is chosen for, latency -- launch, first loads, one pass through the
// ring, the exchange in the cluster -- so the split is taken to give every SM a CTA; for unrolled
// convolutions the producers' issue slots.  The second group halves what a k-block waits for where an SM has
// one CTA (one B200, one group -> two, us: fp32 512 x 128 x 784 16.7 -> 11.5, 600 x 600 x 600 24.5 -> 14.6).
// Unrolled convolutions whose filters were laid out beforehand leave the producers only the gathered rows, and
// tiles of more pixels pay (batch 100, forward / input gradient, us: 16 channels at 32x32 20.2 -> 12.9 / 25.1 ->
// 12.9, 32 at 16x16 14.6 -> 12.1 / 23.3 -> 12.2, 64 at 8x8 14.3 -> 12.1 / 14.2 -> 12.1); the filters' way from L2 to
// every SM, 256 bytes a row and k-block, then bounds the widest tiles.
#ifndef B2_DIRECT_CUH
#define B2_DIRECT_CUH
#include "b2_direct.h"
#include "b2_gemm_impl.cuh"

namespace {

constexpr int kDirThreads = 288;
constexpr int kDirMaxK = 4608;            // columns of the gather table
// groups: producers in groups of eight warps, each with a k-block of its own; more than one only where every
// SM has a single CTA, which then has the shared memory for a deeper ring
__host__ __device__ constexpr int dir_stages(int bn, int groups = 1) {
    return groups > 1 ? (bn >= 64 ? 3 : 4) : bn == 128 ? 3 : 2;
}
__host__ __device__ constexpr int dir_threads(int groups, bool staged = false) { return groups * 256 + (staged ? 64 : 32); }
__host__ __device__ constexpr int dir_stage_bytes(int bn) { return 2 * (128 + bn) * 128; }
__host__ __device__ constexpr int dir_ring_bytes(int bn, int groups = 1) { return dir_stages(bn, groups) * dir_stage_bytes(bn); }
__host__ __device__ constexpr int dir_tmem_cols(int mode, int bn, int pairs = 1) {
    int need = (mode == MODE_FLEX16 ? 3 : 2 * pairs) * bn, c = 32;
    while (c < need) c *= 2;
    return c;
}

// gathered fp32 rows: pairs of sums that the k-blocks go to by turns
__host__ __device__ constexpr int dir_pairs(int bn, int groups) { return bn <= 32 || (bn == 64 && groups > 1) ? 4 : 2; }

__host__ __device__ inline bool filter_tiles(const b2_direct_args& a) { return a.b_kind == B2_OPERAND_FILTER; }

__host__ __device__ inline int dir_table_bytes(const b2_direct_args& a, int columns) {
    return a.a_kind != B2_OPERAND_GATHER ? 0 : columns * (filter_tiles(a) && !a.staged ? 16 : 8);
}

struct DirectParams {
    b2_direct_args a;
    int num_kb, kb_per_split, splits;
    int a_vec, b_vec;                     // 16-byte loads (K contiguous) / row pairs (flex16, others)
};

// a = hi + lo with hi rounded to tf32, ties away from zero: what cvt.rna.tf32 gives for every finite a
// (infinities and NaN end as NaN in the product either way), on the full-rate integer pipe
__device__ __forceinline__ void dir_split_tf32(float a, float& hi, float& lo) {
    hi = __uint_as_float((__float_as_uint(a) + 0x1000u) & 0xffffe000u);
    lo = a - hi;
}
__device__ __forceinline__ unsigned swz(int row, int chunk) {
    return (unsigned)(row * 128 + ((chunk ^ (row & 7)) << 4));
}
// ---- operand tiles ---------------------------------------------------------------------------
// Registers of one thread's share of an operand's k-block, loaded in one go so that all loads are
// in flight together, and stored a k-block later.
//
// fp32, K contiguous: unit = 4 rows x 8 chunks of 16 bytes, a lane holds one chunk; else unit = 32 rows
// x 1 chunk, a lane holds four columns of its row.  flex16: the same with 16 columns to a chunk; with
// rows contiguous a lane takes two neighbouring rows (one 4-byte load brings both).
template <int MODE, int ROWS>
struct OperandTile {
    static constexpr int kUnits = MODE == MODE_FLEX16 ? (ROWS >= 64 ? ROWS / 64 : 1) : (ROWS >= 32 ? ROWS / 32 : 1);
    static constexpr int kRegs = MODE == MODE_FLEX16 ? 16 * kUnits : 4 * kUnits;
    static constexpr int kKUnits = ROWS / 4 >= 8 ? ROWS / 32 : 1;      // units per warp, K contiguous
    unsigned r[kRegs];

    // -- K contiguous: byte offsets of this lane's chunk in each of its rows (-1: no such row)
    __device__ __forceinline__ static void offsets_k(long long (&at)[kKUnits], long long rs, int row0, int rows,
                                                     int warp, int lane) {
        constexpr int per = MODE == MODE_FLEX16 ? 16 : 4, size = MODE == MODE_FLEX16 ? 2 : 4;
#pragma unroll
        for (int i = 0; i < kKUnits; ++i) {
            const int lr = (warp + 8 * i) * 4 + (lane >> 3), row = row0 + lr;
            at[i] = lr < ROWS && row < rows ? ((long long)row * rs + (lane & 7) * per) * size : -1;
        }
    }
    // `left`: columns from k0 to the end of K
    __device__ __forceinline__ void load_k(const void* src, const long long (&at)[kKUnits], int k0, int left,
                                           int vec, int lane) {
        constexpr int per = MODE == MODE_FLEX16 ? 16 : 4, regs = MODE == MODE_FLEX16 ? 8 : 4,
                      size = MODE == MODE_FLEX16 ? 2 : 4;
        const char* base = (const char*)src + (long long)k0 * size;
        const bool whole = vec && (lane & 7) * per + per <= left;
#pragma unroll
        for (int i = 0; i < kKUnits; ++i) {
#pragma unroll
            for (int j = 0; j < regs; ++j) r[regs * i + j] = 0;
            if (at[i] < 0) continue;
            const char* p = base + at[i];
            if (whole) {
                const uint4 a = __ldg((const uint4*)p);
                r[regs * i + 0] = a.x; r[regs * i + 1] = a.y; r[regs * i + 2] = a.z; r[regs * i + 3] = a.w;
                if (MODE == MODE_FLEX16) {
                    const uint4 b = __ldg((const uint4*)p + 1);
                    r[regs * i + regs - 4] = b.x; r[regs * i + regs - 3] = b.y;
                    r[regs * i + regs - 2] = b.z; r[regs * i + regs - 1] = b.w;
                }
            } else {
#pragma unroll
                for (int j = 0; j < per; ++j) {
                    if ((lane & 7) * per + j >= left) continue;
                    if (MODE == MODE_FLEX16)
                        r[regs * i + (j >> 1)] |= (unsigned)((const unsigned short*)p)[j] << ((j & 1) * 16);
                    else
                        r[regs * i + j % regs] = ((const unsigned*)p)[j];
                }
            }
        }
    }
    __device__ __forceinline__ void store_k(unsigned char* p0, unsigned char* p1, int warp, int lane) const {
        const int chunk = lane & 7;
#pragma unroll
        for (int i = 0; i < kKUnits; ++i) {
            const int lr = (warp + 8 * i) * 4 + (lane >> 3);
            if (lr >= ROWS) continue;
            const unsigned at = swz(lr, chunk);
            if (MODE == MODE_FLEX16) {
                const unsigned* w = r + 8 * i;
                uint4 h, l;
                h.x = __byte_perm(w[0], w[1], 0x7531); l.x = __byte_perm(w[0], w[1], 0x6420);
                h.y = __byte_perm(w[2], w[3], 0x7531); l.y = __byte_perm(w[2], w[3], 0x6420);
                h.z = __byte_perm(w[4], w[5], 0x7531); l.z = __byte_perm(w[4], w[5], 0x6420);
                h.w = __byte_perm(w[6], w[7], 0x7531); l.w = __byte_perm(w[6], w[7], 0x6420);
                *(uint4*)(p0 + at) = h;
                *(uint4*)(p1 + at) = l;
            } else {
                store_f4(p0, p1, at, r + 4 * i);
            }
        }
    }
    __device__ __forceinline__ static void store_f4(unsigned char* p0, unsigned char* p1, unsigned at,
                                                    const unsigned* v) {
        float4 h, l;
        dir_split_tf32(__uint_as_float(v[0]), h.x, l.x); dir_split_tf32(__uint_as_float(v[1]), h.y, l.y);
        dir_split_tf32(__uint_as_float(v[2]), h.z, l.z); dir_split_tf32(__uint_as_float(v[3]), h.w, l.w);
        *(float4*)(p0 + at) = h;
        *(float4*)(p1 + at) = l;
    }
    // rows of this lane in a group of 32 (fp32) or 64 (flex16): a pair of rows for flex16.  Four
    // lanes of eight start with the odd row, which keeps the 16-byte stores of a phase apart.
    __device__ __forceinline__ static void store_pair(unsigned char* p0, unsigned char* p1, int lr, int chunk,
                                                      int lane, const unsigned* w) {
        uint4 h[2], l[2];
        unsigned* hp[2] = {(unsigned*)&h[0], (unsigned*)&h[1]};
        unsigned* lp[2] = {(unsigned*)&l[0], (unsigned*)&l[1]};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            // words hold (row | next row << 16) of four columns
            const unsigned a = __byte_perm(w[4 * q], w[4 * q + 1], 0x5140), b = __byte_perm(w[4 * q + 2], w[4 * q + 3], 0x5140);
            const unsigned c = __byte_perm(w[4 * q], w[4 * q + 1], 0x7362), d = __byte_perm(w[4 * q + 2], w[4 * q + 3], 0x7362);
            lp[0][q] = __byte_perm(a, b, 0x5410); hp[0][q] = __byte_perm(a, b, 0x7632);
            lp[1][q] = __byte_perm(c, d, 0x5410); hp[1][q] = __byte_perm(c, d, 0x7632);
        }
        const bool odd = (lane >> 2) & 1;
        const unsigned at0 = swz(lr + (odd ? 1 : 0), chunk), at1 = swz(lr + (odd ? 0 : 1), chunk);
        *(uint4*)(p0 + at0) = odd ? h[1] : h[0];
        *(uint4*)(p0 + at1) = odd ? h[0] : h[1];
        *(uint4*)(p1 + at0) = odd ? l[1] : l[0];
        *(uint4*)(p1 + at1) = odd ? l[0] : l[1];
    }
};

template <int MODE, int BN, int AK, int G, bool STAGED>
__global__ void __launch_bounds__(dir_threads(G, STAGED), (BN == 128 || G > 1 ? 1 : 2))
direct_kernel(const __grid_constant__ DirectParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int NST = dir_stages(BN, G), STAGE = dir_stage_bytes(BN), MMA_WARP = 8 * G;
    constexpr int KB = MODE == MODE_FLEX16 ? 128 : 32;            // columns of a k-block
    constexpr int PER = KB / 8;                                   // columns of a 16-byte chunk
    constexpr int PAIRS = MODE == MODE_F32X3 && AK == B2_OPERAND_GATHER ? dir_pairs(BN, G) : 1;
    constexpr int kCols = dir_tmem_cols(MODE, BN, PAIRS);
    // fp32 matrix products: one accumulator, the three products of a k-step in the order of the plane
    // kernels, slices of whole chains -- the same rounding whichever kernel a size takes (a mask `x > 0`
    // of a value near zero would otherwise change with the dispatch)
    constexpr bool ONE_CHAIN = MODE == MODE_F32X3 && AK != B2_OPERAND_GATHER;
    typedef OperandTile<MODE, 128> ATile;
    typedef OperandTile<MODE, BN> BTile;
    unsigned long long* full_bar = (unsigned long long*)(smem + NST * STAGE);     // [NST]
    unsigned long long* empty_bar = full_bar + NST;                               // [NST]
    unsigned long long* tmem_full = empty_bar + NST;
    unsigned* tmem_holder = (unsigned*)(tmem_full + 1);
    int* fail_flag = (int*)(tmem_holder + 1);
    int2* tab = (int2*)((unsigned char*)full_bar + 128);                          // [K of the slice] gather table
    int2* ftab = tab + p.kb_per_split * KB;                                       // likewise, of the filters
    const bool tiled = AK == B2_OPERAND_GATHER && filter_tiles(p.a);
    const bool ftiled = tiled && !STAGED;                         // the producers make the rows of the filters

    // (warp: within its group of eight)
    const int wid = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31, group = wid >> 3, warp = wid & 7;
    const b2_direct_args& a = p.a;
    const int m0 = blockIdx.y * 128, n0 = blockIdx.x * BN;
    const int rank = blockIdx.z, kb0 = rank * p.kb_per_split;
    const int nkb = min(p.kb_per_split, p.num_kb - kb0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < NST; ++s) { mbar_init(&full_bar[s], STAGED ? 9 : 8); mbar_init(&empty_bar[s], 1); }
        mbar_init(tmem_full, 1);
        *fail_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (wid == MMA_WARP) {
        tmem_alloc(tmem_holder, kCols);
        // the next kernel may start its set-up now: not before this CTA holds its tensor memory, or
        // the two could each wait for what the other has
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    if (AK == B2_OPERAND_GATHER) {
        // offset of every column of this slice and the bit of its tap (none beyond K)
        const b2_gather& g = a.g;
        const int RS = g.R * g.S;
        for (int i = threadIdx.x; i < nkb * KB; i += dir_threads(G, STAGED)) {
            const int k = kb0 * KB + i;
            int2 e = make_int2(0, 0), f = make_int2(0, 0x7fff7fff);       // (no filter has that tap)
            if (k < a.K) {
                const int c = g.channel_last ? k % g.channels : k / RS, rs = g.channel_last ? k / g.channels : k % RS;
                const int r = rs / g.S, s = rs - r * g.S;
                e = make_int2(((c * g.H + r * g.tap_h) * g.W + s * g.tap_w) * g.N, (int)(1u << rs));
                f = make_int2(c * (int)a.b_ks, ((g.f0_h + g.f1_h * r) & 0xffff) << 16 | ((g.f0_w + g.f1_w * s) & 0xffff));
            }
            tab[i] = e;
            if (ftiled) ftab[i] = f;
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = (unsigned)warp_uniform((int)*tmem_holder);

    if (wid < MMA_WARP) {
        // ---- producers
        // fp32 loads a k-block ahead; a flex16 k-block is 128 columns, few of them make a problem, and a
        // second set of registers would spill
        constexpr bool AHEAD = MODE != MODE_FLEX16;
        ATile ta[AHEAD ? 2 : 1];
        BTile tb[AHEAD ? 2 : 1];
        // gathered rows: fixed for the whole CTA.  fp32: one row of a group of 32; flex16: two of 64.
        constexpr int GR = MODE == MODE_FLEX16 ? 2 : 1;
        const int a_lr = MODE == MODE_FLEX16 ? (warp & 1) * 64 + 2 * lane : (warp & 3) * 32 + lane;
        const int a_c0 = MODE == MODE_FLEX16 ? warp >> 1 : warp >> 2;              // first chunk
        constexpr int a_cs = MODE == MODE_FLEX16 ? 4 : 2;                          // chunk step
        constexpr int A_UNITS = 8 / a_cs;                                          // 2 or 4
        const void* a_row[GR];
        unsigned mask[GR];                                                         // bit t: tap t inside
        bool pair = GR == 2 && p.a_vec;
        if (AK != B2_OPERAND_K) {
#pragma unroll
            for (int e = 0; e < GR; ++e) {
                const int row = m0 + a_lr + e;
                mask[e] = 0;
                long long base = row;
                if (AK == B2_OPERAND_GATHER) {
                    const b2_gather& g = a.g;
                    base = 0;
                    if (row < a.M) {
                        const int n = row % g.N, pq = row / g.N, q = pq % g.Q, pp = pq / g.Q;
                        const int h0 = pp * g.step_h + g.off_h, w0 = q * g.step_w + g.off_w;
                        for (int r = 0, t = 0; r < g.R; ++r)
                            for (int s = 0; s < g.S; ++s, ++t) {
                                const int hh = h0 + r * g.tap_h, ww = w0 + s * g.tap_w;
                                if (hh >= 0 && hh < g.H && ww >= 0 && ww < g.W) mask[e] |= 1u << t;
                            }
                        base = ((long long)h0 * g.W + w0) * g.N + n;
                    }
                } else if (row < a.M) {
                    mask[e] = 1u;
                }
                a_row[e] = (const char*)a.A + base * (MODE == MODE_FLEX16 ? 2 : 4);
            }
            if (GR == 2) pair = pair && (mask[GR - 1] == mask[0]) && m0 + a_lr + 1 < a.M;
        }
        long long a_at[ATile::kKUnits], b_at[BTile::kKUnits];
        if (AK == B2_OPERAND_K) ATile::offsets_k(a_at, a.a_rs, m0, a.M, warp, lane);
        if (!STAGED) BTile::offsets_k(b_at, a.b_rs, n0, a.N, warp, lane);
        // filter rows of this lane: channel's place in the filters and the pixel's share of the tap
        constexpr int FR = BTile::kUnits * GR;
        int f_at[FR], f_h[FR], f_w[FR];
        if (AK == B2_OPERAND_GATHER && ftiled) {
            const b2_gather& g = a.g;
#pragma unroll
            for (int i = 0; i < FR; ++i) {
                const int lr = (i / GR) * 32 * GR + GR * lane + i % GR, row = n0 + lr, pix = row / g.kt;
                const int gy = pix / g.gw, gx = pix - gy * g.gw;
                f_at[i] = (row - pix * g.kt) * (int)a.b_rs;
                f_h[i] = lr < BN && row < a.N ? g.f2_h * gy : 1 << 20;
                f_w[i] = g.f2_w * gx;
            }
        }
        auto load = [&](int kb, ATile& A, BTile& B) {
            const int kt = kb * KB, k0 = kb0 * KB + kt;
            if (AK == B2_OPERAND_K) {
                A.load_k(a.A, a_at, k0, a.K - k0, p.a_vec, lane);
            } else {
#pragma unroll
                for (int i = 0; i < A_UNITS; ++i) {
                    const int kc = (a_c0 + a_cs * i) * PER;
                    int4 pair_of;
#pragma unroll
                    for (int j = 0; j < PER; ++j) {
                        unsigned v = 0;
                        long long o;
                        bool in0, in1 = false;
                        if (AK == B2_OPERAND_GATHER) {
                            // two entries to a load
                            if (j % 2 == 0) pair_of = *(const int4*)(tab + kt + kc + j);
                            const int2 t = j % 2 == 0 ? make_int2(pair_of.x, pair_of.y) : make_int2(pair_of.z, pair_of.w);
                            o = t.x;
                            in0 = (mask[0] & (unsigned)t.y) != 0;
                            if (GR == 2) in1 = (mask[GR - 1] & (unsigned)t.y) != 0;
                        } else {
                            o = (long long)(k0 + kc + j) * a.a_ks;
                            in0 = mask[0] && k0 + kc + j < a.K;
                            if (GR == 2) in1 = mask[GR - 1] && k0 + kc + j < a.K;
                        }
                        if (MODE == MODE_FLEX16) {
                            if (pair) {
                                if (in0) v = __ldg((const unsigned*)((const short*)a_row[0] + o));
                            } else {
                                if (in0) v = __ldg((const unsigned short*)a_row[0] + o);
                                if (in1) v |= (unsigned)__ldg((const unsigned short*)a_row[GR - 1] + o) << 16;
                            }
                        } else if (in0) {
                            v = __float_as_uint(__ldg((const float*)a_row[0] + o));
                        }
                        A.r[PER * i + j] = v;
                    }
                }
            }
            if (STAGED) {
                // (the copying warp brings B)
            } else if (AK == B2_OPERAND_GATHER && ftiled) {
                const b2_gather& g = a.g;
                const int mult = (int)(g.channel_last ? a.g.channels : g.kt);     // filters: tap stride
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    const int2 f = ftab[kt + warp * PER + j];
                    const int th = f.y >> 16, tw = (short)f.y;
#pragma unroll
                    for (int i = 0; i < BTile::kUnits; ++i) {
                        unsigned v = 0;
#pragma unroll
                        for (int e = 0; e < GR; ++e) {
                            const int r = th + f_h[i * GR + e], s = tw + f_w[i * GR + e];
                            if ((unsigned)r >= (unsigned)g.fr || (unsigned)s >= (unsigned)g.fs) continue;
                            const int at = f.x + f_at[i * GR + e] + (r * g.fs + s) * mult;
                            if (MODE == MODE_FLEX16) v |= (unsigned)__ldg((const unsigned short*)a.B + at) << (16 * e);
                            else v = __float_as_uint(__ldg((const float*)a.B + at));
                        }
                        B.r[PER * i + j] = v;
                    }
                }
            } else if (a.b_kind == B2_OPERAND_K) {
                B.load_k(a.B, b_at, k0, a.K - k0, p.b_vec, lane);
            } else {
                // chunk = warp, groups of 32 (64) rows
                const bool whole = k0 + KB <= a.K;
                const char* from = (const char*)a.B + (n0 + lane + (long long)(k0 + warp * PER) * a.b_ks) * 4;
#pragma unroll
                for (int i = 0; i < BTile::kUnits; ++i) {
                    if (MODE != MODE_FLEX16) {
                        const bool there = i * 32 + lane < BN && n0 + i * 32 + lane < a.N;
                        const float* s = (const float*)from + i * 32;
#pragma unroll
                        for (int j = 0; j < PER; ++j, s += a.b_ks)
                            B.r[PER * i + j] = there && (whole || k0 + warp * PER + j < a.K) ? __float_as_uint(__ldg(s)) : 0u;
                        continue;
                    }
                    const int lr = i * 64 + 2 * lane, row = n0 + lr;
                    const bool in0 = lr < BN && row < a.N, in1 = lr + 1 < BN && row + 1 < a.N;
#pragma unroll
                    for (int j = 0; j < PER; ++j) {
                        const int k = k0 + warp * PER + j;
                        unsigned v = 0;
                        if (k < a.K) {
                            const unsigned short* s = (const unsigned short*)a.B + row + (long long)k * a.b_ks;
                            if (p.b_vec && in1) v = __ldg((const unsigned*)s);
                            else {
                                if (in0) v = __ldg(s);
                                if (in1) v |= (unsigned)__ldg(s + 1) << 16;
                            }
                        }
                        B.r[PER * i + j] = v;
                    }
                }
            }
        };
        auto store = [&](int s, const ATile& A, const BTile& B) {
            unsigned char* st = smem + s * STAGE;
            unsigned char* b0 = st + 2 * 128 * 128;
            if (AK == B2_OPERAND_K) {
                A.store_k(st, st + 128 * 128, warp, lane);
            } else {
#pragma unroll
                for (int i = 0; i < A_UNITS; ++i) {
                    if (MODE == MODE_FLEX16)
                        ATile::store_pair(st, st + 128 * 128, a_lr, a_c0 + a_cs * i, lane, A.r + PER * i);
                    else
                        ATile::store_f4(st, st + 128 * 128, swz(a_lr, a_c0 + a_cs * i), A.r + PER * i);
                }
            }
            if (STAGED) {
            } else if (a.b_kind == B2_OPERAND_K) {
                B.store_k(b0, b0 + BN * 128, warp, lane);
            } else {
#pragma unroll
                for (int i = 0; i < BTile::kUnits; ++i) {
                    const int lr = MODE == MODE_FLEX16 ? i * 64 + 2 * lane : i * 32 + lane;
                    if (lr >= BN) continue;
                    if (MODE == MODE_FLEX16) BTile::store_pair(b0, b0 + BN * 128, lr, warp, lane, B.r + PER * i);
                    else BTile::store_f4(b0, b0 + BN * 128, swz(lr, warp), B.r + PER * i);
                }
            }
        };
        if (AHEAD && group < nkb) load(group, ta[0], tb[0]);
        int s = group % NST;
        unsigned parity = 1;
        bool ok = true;
        auto put = [&](int kb, ATile& A, BTile& B, ATile& An, BTile& Bn) {
            if (!AHEAD) load(kb, A, B);
            else if (kb + G < nkb) load(kb + G, An, Bn);          // in flight while this one is stored
            if (ok && !mbar_wait(&empty_bar[s], parity)) { atomicExch(fail_flag, 1); ok = false; }
            store(s, A, B);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_bar[s]);
            s += G;
            if (s >= NST) { s -= NST; parity ^= 1u; }
        };
        constexpr int kNext = AHEAD ? 1 : 0;
        for (int kb = group; kb < nkb; kb += 2 * G) {
            put(kb, ta[0], tb[0], ta[kNext], tb[kNext]);
            if (kb + G < nkb) put(kb + G, ta[kNext], tb[kNext], ta[0], tb[0]);
        }
    } else if (STAGED && wid > MMA_WARP) {
        if (elect_one()) {
            // ---- copies of B: one to a k-block, in the order of n tiles and k-blocks
            constexpr unsigned bytes = 2 * BN * 128;
            const char* src = (const char*)a.staged + ((long long)blockIdx.x * p.num_kb + kb0) * bytes;
            int s = 0, n = 0;
            unsigned parity = 1;
            for (; n < nkb; ++n) {
                if (!mbar_wait(&empty_bar[s], parity)) { atomicExch(fail_flag, 1); break; }
                mbar_expect_tx(&full_bar[s], bytes);
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                    ::"r"(smem_u32(smem + s * STAGE + 2 * 128 * 128)), "l"(src + (long long)n * bytes), "r"(bytes),
                      "r"(smem_u32(&full_bar[s])) : "memory");
                if (++s == NST) { s = 0; parity ^= 1u; }
            }
            // what is in flight lands before the block ends, whatever has become of the other roles
            for (int i = n > NST ? n - NST : 0; i < n; ++i)
                if (!mbar_wait(&full_bar[i % NST], (i / NST) & 1)) { atomicExch(fail_flag, 1); break; }
        }
    } else if (elect_one()) {
        // ---- MMA issue
        const unsigned id_ss = make_idesc(2, 1, 1, BN), id_su = make_idesc(2, 1, 0, BN),
                       id_us = make_idesc(2, 0, 1, BN), id_uu = make_idesc(2, 0, 0, BN);
        const unsigned id_t1 = make_idesc(1, 2, 2, BN), id_t2 = make_idesc(1, 2, 2, 2 * BN);
        int s = 0;
        unsigned parity = 0;
        for (int kb = 0; kb < nkb; ++kb) {
            if (!mbar_wait(&full_bar[s], parity)) { atomicExch(fail_flag, 1); break; }
            tc_fence_after();
            unsigned char* st = smem + s * STAGE;
            const unsigned long long dA0 = make_smem_desc(st), dA1 = make_smem_desc(st + 128 * 128);
            const unsigned long long dB0 = make_smem_desc(st + 2 * 128 * 128);
            const unsigned long long dB1 = make_smem_desc(st + 2 * 128 * 128 + BN * 128);
            const unsigned sums = tmem_base + kb % PAIRS * 2 * BN;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const unsigned long long adv = (unsigned long long)(2 * k);
                const unsigned acc = (kb >= PAIRS || k > 0) ? 1u : 0u;
                if (MODE == MODE_FLEX16) {
                    tc_mma<MODE>(tmem_base, dA0 + adv, dB0 + adv, id_ss, acc);               // HH
                    tc_mma<MODE>(tmem_base + BN, dA0 + adv, dB1 + adv, id_su, acc);          // X += ah*bl
                    tc_mma<MODE>(tmem_base + BN, dA1 + adv, dB0 + adv, id_us, 1u);           // X += al*bh
                    tc_mma<MODE>(tmem_base + 2 * BN, dA1 + adv, dB1 + adv, id_uu, acc);      // LL
                } else if (ONE_CHAIN) {
                    tc_mma<MODE>(tmem_base, dA0 + adv, dB0 + adv, id_t1, acc);               // hi*hi
                    tc_mma<MODE>(tmem_base, a.colmajor ? dA1 + adv : dA0 + adv,
                                 a.colmajor ? dB0 + adv : dB1 + adv, id_t1, 1u);
                    tc_mma<MODE>(tmem_base, a.colmajor ? dA0 + adv : dA1 + adv,
                                 a.colmajor ? dB1 + adv : dB0 + adv, id_t1, 1u);
                } else {
                    tc_mma<MODE>(sums, dA0 + adv, dB0 + adv, id_t2, acc);                    // hh | x
                    tc_mma<MODE>(sums + BN, dA1 + adv, dB0 + adv, id_t1, 1u);                // x += lo*hi
                }
            }
            tc_commit(&empty_bar[s]);
            if (++s == NST) { s = 0; parity ^= 1u; }
        }
        tc_commit(tmem_full);
    }
    __syncwarp();

    // ---- epilogue: warps 0-7, lane quarter = warp % 4, the two warps of a quarter take the 8-column
    // pieces in turn
    typedef typename std::conditional<MODE == MODE_FLEX16, long long, float>::type Sum;
    Sum* red = (Sum*)smem;                                        // [BN][128], slices only
    const int quarter = warp & 3, half = warp >> 2;
    const int lrow = quarter * 32 + lane, row = m0 + lrow;
    const int splits = p.splits;
    bool ok = true;
    int stat = 0;
    unsigned long long pmax = 0;
    int sh = 0;
    if (MODE == MODE_FLEX16 && wid < 8) {
        const float q_out = a.probe ? 1.0f : a.table[a.slotC].inv_scale;
        sh = -ilogbf(a.table[a.slotA].scale * a.table[a.slotB].scale * q_out);
    }
    // tiles of several pixels: where the row's tile starts
    int tile_p = 0, tile_q = 0;
    long long tile_at = 0;
    if (tiled) {
        const int n = row % a.g.N, pq = row / a.g.N;
        tile_p = pq / a.g.Q * a.g.gh; tile_q = pq % a.g.Q * a.g.gw;
        tile_at = ((long long)tile_p * a.g.out_q + tile_q) * a.g.N + n;
    }
    auto finish = [&](int c0, Sum* v) {
        // eight results of one row: tail, rescale, statistics, store
        if (row >= a.M) return;
        int col = n0 + c0;
        const int live = a.N - col;
        long long at = a.colmajor ? (long long)col * a.ldc + row : (long long)row * a.ldc + col;
        if (tiled) {
            const int pix = col / a.g.kt, gy = pix / a.g.gw, gx = pix - gy * a.g.gw;
            col -= pix * a.g.kt;
            if (tile_p + gy >= a.g.out_p || tile_q + gx >= a.g.out_q) return;
            at = (long long)col * a.ldc + tile_at + ((long long)gy * a.g.out_q + gx) * a.g.N;
        }
        const long long dc = a.colmajor ? a.ldc : 1;
        if (MODE == MODE_FLEX16) {
            int q[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                q[j] = 0;
                if (j >= live) continue;
                const long long x = (long long)v[j];
                if (a.probe) {
                    const unsigned long long m = (unsigned long long)(x < 0 ? -x : x);
                    pmax = m > pmax ? m : pmax;
                } else {
                    q[j] = rescale_i64(x, sh);
                    const int m = q[j] < 0 ? -q[j] : q[j];
                    stat = m > stat ? m : stat;
                }
            }
            if (a.probe) return;
            short* out = (short*)a.C + at;
            if (!a.colmajor && live >= 8 && ((uintptr_t)out & 15) == 0) {
                uint4 w;
                w.x = (q[0] & 0xffff) | (q[1] << 16); w.y = (q[2] & 0xffff) | (q[3] << 16);
                w.z = (q[4] & 0xffff) | (q[5] << 16); w.w = (q[6] & 0xffff) | (q[7] << 16);
                *(uint4*)out = w;
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j < live) out[j * dc] = (short)q[j];
            }
        } else {
            // (one uniform branch per operand, its eight loads together)
            float y[8], t[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) y[j] = (float)v[j];
            auto fetch = [&](const float* x, long long step) {
#pragma unroll
                for (int j = 0; j < 8; ++j) t[j] = j < live ? __ldg(x + j * step) : 0.0f;
            };
            if (a.bias) {
                fetch(a.bias + col, 1);
#pragma unroll
                for (int j = 0; j < 8; ++j) y[j] += t[j];
            }
            if (a.residual) {
                fetch(a.residual + at, dc);
#pragma unroll
                for (int j = 0; j < 8; ++j) y[j] += t[j];
            }
            if (a.relu) {
#pragma unroll
                for (int j = 0; j < 8; ++j) y[j] = y[j] < 0.0f ? 0.0f : y[j];      // (keeps NaN, as max(x, 0) does)
            }
            if (a.mask) {
                fetch(a.mask + at, dc);
#pragma unroll
                for (int j = 0; j < 8; ++j) y[j] *= t[j] > 0.0f ? 1.0f : 0.0f;     // (likewise)
            }
            float* out = (float*)a.C + at;
            if (!a.colmajor && live >= 8 && ((uintptr_t)out & 15) == 0) {
                *(float4*)out = make_float4(y[0], y[1], y[2], y[3]);
                *(float4*)(out + 4) = make_float4(y[4], y[5], y[6], y[7]);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j < live) out[j * dc] = y[j];
            }
        }
    };
    if (wid < 8) {
        ok = mbar_wait(tmem_full, 0);
        if (!ok) atomicExch(fail_flag, 1);
        tc_fence_after();
        const unsigned lane_addr = tmem_base + ((unsigned)(quarter * 32) << 16);
        for (int c0 = half * 8; c0 < BN; c0 += 16) {
            if (n0 + c0 >= a.N) break;
            Sum v[8];
            if (MODE == MODE_FLEX16) {
                unsigned hh[8], xx[8], ll[8];
                tmem_ld8(lane_addr + c0, hh);
                tmem_ld8(lane_addr + BN + c0, xx);
                tmem_ld8(lane_addr + 2 * BN + c0, ll);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    v[j] = (Sum)(((long long)(int)hh[j] << 16) + ((long long)(int)xx[j] << 8) + (long long)(int)ll[j]);
            } else {
                unsigned hh[8], xx[8];
                tmem_ld8(lane_addr + c0, hh);
                if (!ONE_CHAIN) tmem_ld8(lane_addr + BN + c0, xx);
                tmem_ld_wait();
#pragma unroll
                for (int q = 1; q < PAIRS; ++q) {
                    if (q >= nkb) break;
                    unsigned h[8], x[8];
                    tmem_ld8(lane_addr + q * 2 * BN + c0, h);
                    tmem_ld8(lane_addr + q * 2 * BN + BN + c0, x);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        hh[j] = __float_as_uint(__uint_as_float(hh[j]) + __uint_as_float(h[j]));
                        xx[j] = __float_as_uint(__uint_as_float(xx[j]) + __uint_as_float(x[j]));
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    v[j] = ONE_CHAIN ? (Sum)__uint_as_float(hh[j])
                                     : (Sum)(__uint_as_float(hh[j]) + __uint_as_float(xx[j]));
            }
            if (splits == 1) {
                if (ok) finish(c0, v);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) red[(c0 + j) * 128 + lrow] = v[j];
            }
        }
    }
    if (splits > 1) {
        cluster_sync();
        if (wid < 8) {
            // this CTA's share of the pieces: every splits-th, dealt to the warps of a quarter
            for (int c0 = (rank + half * splits) * 8; c0 < BN; c0 += 16 * splits) {
                if (n0 + c0 >= a.N) break;
                Sum v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = 0;
                // (a peer's values take about 700 cycles: those of several slices come together)
                constexpr int Z = MODE == MODE_FLEX16 ? 2 : 4;
                for (int z0 = 0; z0 < splits; z0 += Z) {
                    Sum t[Z][8];
#pragma unroll
                    for (int z = 0; z < Z; ++z) {
                        if (z0 + z >= splits) break;
                        const unsigned at = map_rank(red + c0 * 128 + lrow, z0 + z);
#pragma unroll
                        for (int j = 0; j < 8; ++j) t[z][j] = ld_peer(at + j * 128 * (unsigned)sizeof(Sum), (Sum)0);
                    }
#pragma unroll
                    for (int z = 0; z < Z; ++z) {
                        if (z0 + z >= splits) break;
#pragma unroll
                        for (int j = 0; j < 8; ++j) v[j] += t[z][j];
                    }
                }
                if (ok) finish(c0, v);
            }
        }
        cluster_sync();                                           // peers may still be reading
    }
    if (MODE == MODE_FLEX16 && wid < 8) {
        if (a.probe) {
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long t = __shfl_xor_sync(0xffffffffu, pmax, o);
                pmax = t > pmax ? t : pmax;
            }
            if (lane == 0 && pmax) atomicMax(a.probe_out, pmax);
        } else {
            for (int o = 16; o > 0; o >>= 1) {
                const int t = __shfl_xor_sync(0xffffffffu, stat, o);
                stat = t > stat ? t : stat;
            }
            if (lane == 0 && stat) atomicMax(a.stats + a.slotC, stat);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (wid == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kCols);
    }
    if (threadIdx.x == 0 && *fail_flag && a.status) atomicExch(a.status, 1);
}

// ---- host ------------------------------------------------------------------------------------
struct DirectShape { int bn, splits, kb_per_split, waves, groups; long long cost; };

// `plain`: the shape of a kernel with one group of producers and one pair of sums, for what it adds up in
// one go (see b2_direct_args::longest).
template <int MODE>
DirectShape direct_shape(const b2_direct_args& a, bool plain = false) {
    const int KB = MODE == MODE_FLEX16 ? 128 : 32;
    const int num_kb = (a.K + KB - 1) / KB;
    // fp32: 16 k-blocks to a chain; flex16: exact int32 sums up to 32768 columns
    const int most = MODE == MODE_FLEX16 ? 256 : 16;
    DirectShape best = {0, 0, 0, 0, 1, -1};
    const long long tm = (a.M + 127) / 128;
    int per_of[9] = {};                                           // k-blocks of a slice, 0: not so many slices
    for (int want = 1; want <= 8 && want <= num_kb; ++want) {
        const bool chains = MODE == MODE_F32X3 && a.a_kind != B2_OPERAND_GATHER && want > 1;
        const int per = chains ? most : (num_kb + want - 1) / want;
        if ((num_kb + per - 1) / per == want && per <= most) per_of[want] = per;
    }
    for (int bn = 16; bn <= 128; bn *= 2) {
        if (bn > 16 && bn / 2 >= a.N) break;
        const long long tiles = tm * ((a.N + bn - 1) / bn);
        for (int splits = 1; splits <= 8; ++splits) {
            const int per = per_of[splits];
            if (!per) continue;
            const int tab = dir_table_bytes(a, per * KB);
            if (1152 + dir_ring_bytes(bn) + tab > 232448) continue;
            // Measured on one B200 (cycles at 1.9 GHz): the producers set the pace, 7 (fp32) or 22
            // (flex16) cycles an operand row of a k-block when they keep an SM busy, and a k-block
            // takes 1000 + 6 bn (gathered 2000 to 3500) or 4000 cycles from load to commit when they do
            // not; the two CTAs of an SM overlap.  Gathered rows cost their address and bounds, filters as
            // a tile's pixels see them the same, more where the lanes' rows lie apart; slices of their wide
            // tiles 15000 more.
            // Rows along K that do not start on 16-byte boundaries are loaded value by value: twice (flex16)
            // and 1.5 times (fp32) the producers' instructions, and 6000 cycles a k-block at the least.
            const int vec = MODE == MODE_FLEX16 ? 8 : 4;
            const bool a_single = a.a_kind == B2_OPERAND_K && a.a_rs % vec != 0;
            const bool b_single = a.b_kind == B2_OPERAND_K && a.b_rs % vec != 0;
            const double single = MODE == MODE_FLEX16 ? 2.0 : 1.5;
            const double ra = a.a_kind == B2_OPERAND_GATHER ? (a.staged ? 1.25 : 1.5) : a_single ? single : 1.0;
            const double rb = a.staged ? 0.0 : filter_tiles(a) ? (a.g.channel_last ? 3.5 : 1.5) : b_single ? single : 1.0;
            const long long pace = (long long)((128 * ra + bn * rb) * (MODE == MODE_FLEX16 ? (bn == 128 ? 33 : 22) : 7));
            const long long lat = MODE == MODE_FLEX16 ? (a_single || b_single ? 6000 : 4000)
                                  : a.a_kind != B2_OPERAND_GATHER ? 1000 + 6 * bn
                                  : a.staged ? (bn == 128 ? 1500 : 1700 + 6 * bn) : bn >= 64 ? 3500 : 1600 + 25 * bn;
            // staged filters: 256 bytes a row and k-block from L2 to every SM (128 rows: 1580 cycles with one
            // group of producers or two)
            const long long copies = a.staged ? 25 * bn / 2 : 0;
            const long long ctas = tiles * splits, per_sm = bn == 128 || 1152 + dir_ring_bytes(bn) + tab > 115000 ? 1 : 2;
            const long long together = ctas <= 148 ? 1 : per_sm;
            // Two groups of producers where each SM has one CTA anyway and a k-block for both: a k-block then
            // takes 65 % (flex16) or 60 % of the cycles (fp32 512 x 128 x 512: 1470 -> 820).  With more CTAs than
            // SMs two of them on an SM do the same (flex16 1500 x 200 x 900 in 144 CTAs of two groups, clusters
            // of three, where 135 find an SM: 26.4 us, 22.5 with one group).  Tiles of 128 columns would spill.
            const int groups = !plain && ctas <= kClusterCtas[splits] && per > 1 && bn < 128 &&
                               1152 + dir_ring_bytes(bn, 2) + tab <= 232448 ? 2 : 1;
            if (a.longest > 0 && !plain && (per + dir_pairs(bn, groups) - 1) / dir_pairs(bn, groups) > a.longest) continue;
            long long kb = together * pace > lat ? together * pace : lat;
            if (groups == 2) kb = kb * (MODE == MODE_FLEX16 ? 65 : 60) / 100;
            if (kb < together * copies) kb = together * copies;
            const long long slots = (long long)kClusterCtas[splits] * (groups == 2 ? 1 : per_sm);
            // (the exchange of slices: 700 and 500 a slice)
            const long long one = 7000 + per * kb + together * bn * (splits > 1 ? 24 : 12) +
                                  (splits == 1 ? 0 : filter_tiles(a) && !a.staged ? 18000 : plain ? 3000 : 700 + 500 * splits);
            if (best.cost >= 0 && one >= best.cost) continue;
            const long long waves = (ctas + slots - 1) / slots, cost = waves * one;
            if (best.cost < 0 || cost < best.cost) best = {bn, splits, per, (int)waves, groups, cost};
        }
    }
    return best;
}

template <int MODE, int BN, int AK, int G, bool STAGED = false>
int direct_launch_as(const DirectParams& p, cudaStream_t st) {
    const int KB = MODE == MODE_FLEX16 ? 128 : 32;
    const int ring = dir_ring_bytes(BN, G);
    static_assert(dir_ring_bytes(BN, G) >= BN * 128 * 8, "the slices' sums are exchanged through the ring");
    const int smem = 1024 + ring + 128 + dir_table_bytes(p.a, p.kb_per_split * KB);
    static bool attr_set = false;
    if (!attr_set) {
        B2_CUDA(cudaFuncSetAttribute(direct_kernel<MODE, BN, AK, G, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     AK == B2_OPERAND_GATHER ? 232448 : 1024 + ring + 128));
        attr_set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.a.N + BN - 1) / BN, (p.a.M + 127) / 128, p.splits);
    cfg.blockDim = dim3(dir_threads(G, STAGED));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = p.splits;
    cfg.attrs = attr;
    cfg.numAttrs = p.splits > 1 ? 2 : 1;
    B2_CUDA(cudaLaunchKernelEx(&cfg, direct_kernel<MODE, BN, AK, G, STAGED>, p));
    return B2_OK;
}

template <int MODE, int BN, int G>
int direct_launch_bn(const DirectParams& p, cudaStream_t st) {
    if constexpr (MODE == MODE_F32X3)
        if (p.a.staged) return direct_launch_as<MODE, BN, B2_OPERAND_GATHER, G, true>(p, st);
    // (flex16 matrix products of several k-blocks come here with both operands along K)
    if constexpr (MODE == MODE_FLEX16 && G > 1) {
        B2_REQUIRE(p.a.a_kind != B2_OPERAND_ROWS, "a product of several k-blocks");
        if (p.a.a_kind == B2_OPERAND_K) return direct_launch_as<MODE, BN, B2_OPERAND_K, G>(p, st);
        return direct_launch_as<MODE, BN, B2_OPERAND_GATHER, G>(p, st);
    }
    switch (p.a.a_kind) {
        case B2_OPERAND_K: return direct_launch_as<MODE, BN, B2_OPERAND_K, G>(p, st);
        case B2_OPERAND_ROWS: return direct_launch_as<MODE, BN, B2_OPERAND_ROWS, G>(p, st);
        default: return direct_launch_as<MODE, BN, B2_OPERAND_GATHER, G>(p, st);
    }
}

template <int MODE>
int direct_launch_mode(const b2_direct_args& a, cudaStream_t st) {
    const DirectShape s = direct_shape<MODE>(a);
    B2_REQUIRE(s.cost >= 0, "K is too long for this kernel");
    B2_REQUIRE(!a.staged || (MODE == MODE_F32X3 && a.a_kind == B2_OPERAND_GATHER && ((uintptr_t)a.staged & 127) == 0),
               "staged filters: of gathered fp32 products, on 128-byte boundaries");
    DirectParams p;
    p.a = a;
    const int KB = MODE == MODE_FLEX16 ? 128 : 32, vec = MODE == MODE_FLEX16 ? 8 : 4;
    p.num_kb = (a.K + KB - 1) / KB;
    p.kb_per_split = s.kb_per_split;
    p.splits = s.splits;
    auto aligned = [&](int kind, const void* x, long long rs, long long ks) {
        if (kind == B2_OPERAND_K) return ((uintptr_t)x & 15) == 0 && rs % vec == 0;
        if (kind == B2_OPERAND_ROWS) return ((uintptr_t)x & 3) == 0 && ks % 2 == 0;
        return ((uintptr_t)x & 3) == 0 && a.g.N % 2 == 0;         // pairs of images of one pixel
    };
    p.a_vec = aligned(a.a_kind, a.A, a.a_rs, a.a_ks);
    p.b_vec = a.b_kind != B2_OPERAND_FILTER && aligned(a.b_kind, a.B, a.b_rs, a.b_ks);
    if (s.groups == 2) {
        switch (s.bn) {
            case 16: return direct_launch_bn<MODE, 16, 2>(p, st);
            case 32: return direct_launch_bn<MODE, 32, 2>(p, st);
            default: return direct_launch_bn<MODE, 64, 2>(p, st);
        }
    }
    switch (s.bn) {
        case 16: return direct_launch_bn<MODE, 16, 1>(p, st);
        case 32: return direct_launch_bn<MODE, 32, 1>(p, st);
        case 64: return direct_launch_bn<MODE, 64, 1>(p, st);
        default: return direct_launch_bn<MODE, 128, 1>(p, st);
    }
}

}  // namespace
#endif  // B2_DIRECT_CUH
