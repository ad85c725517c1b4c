// Convolutions as gathered products, fp32, with the filters laid out beforehand: O^T = Icol * F^T in one launch, the
// rows of Icol (a tile's pixels of one image) gathered on the way in, A's planes in tensor memory (b2_stream.cuh has
// the same for matrix products, b2_direct.cuh the rows of the columns' table and what a tile is).
//
// One CTA per 128 x BN tile (times a slice of K), 864 threads:
//   eight warps copy a k-block's 32 columns: 128 rows each, sixteen bytes a copy (four images of a pixel: other numbers
//             of images stay with b2_direct.cuh; four bytes a copy where the tensor does not start on sixteen), zeros
//             where the tap lies outside; in two groups that take the k-blocks by turns;
//   two groups of eight warps convert, the k-blocks by turns: a lane is a row, a warp has half of its columns, converted
//             by the time the slot in tensor memory is free; afterwards all sixteen are the epilogue (bias, residual,
//             ReLU, mask);
//   one warp copies B's k-blocks as they were laid out, one or two issue the MMAs (by turns: a k-block is a chain of
//             about a thousand cycles for who waits for it and issues it, whatever its size).
// Sums: A_hi x [B_hi | B_lo] -> [hh | x], A_lo x B_hi -> x.  The tensor core's sum loses bits with every k-block, so
// the k-blocks go by turns to two or four hh, added to nearest at the end.  Two of an issuer's share their x between
// them, which holds products 2^-11 of hh's and loses that much less: [hh | x | hh]; for every other k-block of an issuer
// the planes lie in the other order, [B_lo | B_hi] -> [x | hh].  (Against 64 bits: see conv_goes_staged.)
//
// What bounds it: chains of instructions.  Start and first columns 4400 cycles, a k-block 700 to 1000 (a slot of tensor
// memory is filled, announced, multiplied and given back in 1400, there are two or three), the epilogue 2000 for eight
// columns of a warp; without any loads of A or B the launches take 0.89 of their time, with a quarter of the MMAs 0.90.
// One B200, fp32 ResNet-20, kernels of b2_direct.cuh -> this one, us: 22 layers at batch 100 266 -> 239, forward and
// input gradients at batch 256 1000 -> 875; of its epilogue the one with a branch a term took 1.4 times as long in
// training.
#include "b2_stream.cuh"

namespace {

constexpr int kGatThreads = 864;
constexpr int kGatLine = 528;                                       // a column of a raw stage (str_line)
constexpr int kGatRaw = 32 * kGatLine;

// issuers, with two hh and an x each where tensor memory has room
__host__ __device__ constexpr int gat_issuers(int bn) { return bn >= 96 ? 1 : 2; }
__host__ __device__ constexpr int gat_sums(int bn) { return 2 * gat_issuers(bn); }
__host__ __device__ constexpr int gat_group(int bn) { return 3 * bn; }                         // columns of an issuer
// (multiples of the issuers: each waits at barriers of its own)
__host__ __device__ constexpr int gat_slots(int bn) { return bn == 96 ? 3 : bn >= 64 ? 2 : 4; }
__host__ __device__ constexpr int gat_b_stages(int bn) { return bn >= 96 ? 3 : 4; }
constexpr int kGatRawStages = 5;
__host__ __device__ constexpr int gat_tmem(int bn) {
    int need = gat_slots(bn) * 64 + gat_issuers(bn) * gat_group(bn), c = 32;
    while (c < need) c *= 2;
    return c;
}

// x / d for 0 <= x < 2^31: the estimate is one too large at the most
struct Divisor { unsigned d, m; };
inline Divisor divisor(int d) { return {(unsigned)d, (unsigned)((0xffffffffULL + d) / d)}; }
__device__ __forceinline__ int quotient(const Divisor& f, int x) {
    if (f.d == 1) return x;
    const int q = (int)__umulhi((unsigned)x, f.m);
    return (unsigned)q * f.d > (unsigned)x ? q - 1 : q;
}

struct GatherParams {
    b2_direct_args a;
    int num_kb, kb_per_split, splits;
    Divisor taps, tap_cols, channels, images, cols, pixel, pixel_cols;     // R*S, S, channels, N, Q, kt, gw
};

__device__ __forceinline__ void cp_async4(unsigned dst, const void* src, int valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
}

// WIDE: sixteen bytes a copy
template <int BN, bool WIDE>
__global__ void __launch_bounds__(kGatThreads, 1)
gather_kernel(const __grid_constant__ GatherParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int MODE = MODE_F32X3, SLOTS = gat_slots(BN), ISSUERS = gat_issuers(BN), NB = gat_b_stages(BN), NR = kGatRawStages;
    constexpr int PLANES = 2 * BN * 128, COPY_GROUPS = 2, GROUPS = 2;
    unsigned char* planes = smem;                                                 // [NB][first, second][BN][128]
    unsigned char* ring = smem + NB * PLANES;                                     // [NR][32 columns]
    int2* tab = (int2*)(ring + NR * kGatRaw);                                     // [K of the slice] column: offset, tap
    __shared__ unsigned long long raw_full[GROUPS][NR], raw_empty[COPY_GROUPS][NR], slot_full[SLOTS], slot_empty[SLOTS];
    __shared__ unsigned long long b_full[NB], b_empty[NB], sums_full;
    __shared__ unsigned tmem_holder;
    __shared__ int fail_flag;
    __shared__ float bias[BN];

    const int wid = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const b2_direct_args& a = p.a;
    const b2_gather& g = a.g;
    const int m0 = blockIdx.y * 128, n0 = blockIdx.x * BN;
    const int rank = blockIdx.z, kb0 = rank * p.kb_per_split;
    const int nkb = min(p.kb_per_split, p.num_kb - kb0);

    if (threadIdx.x < NR * GROUPS) {
        mbar_init(&raw_full[0][0] + threadIdx.x, 256 / COPY_GROUPS);
        mbar_init(&raw_empty[0][0] + threadIdx.x, 8);
        // (a slot's, not a group's: issuer and converters may be two of a group's k-blocks apart.  With three slots the
        // groups fill one by turns: that the slot before it was free says that this one's phase before is over.)
        if (threadIdx.x < SLOTS) { mbar_init(&slot_full[threadIdx.x], 8); mbar_init(&slot_empty[threadIdx.x], 1); }
        if (threadIdx.x < NB) { mbar_init(&b_full[threadIdx.x], 1); mbar_init(&b_empty[threadIdx.x], 1); }
        if (threadIdx.x == 0) { mbar_init(&sums_full, ISSUERS); fail_flag = 0; }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (wid == 24) {
        tmem_alloc(&tmem_holder, gat_tmem(BN));
        // (not before this CTA holds its tensor memory, or it and the next kernel's could each wait for what the
        // other has)
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    {
        // offset of every column of this slice and the bit of its tap (none beyond K)
        for (int i = threadIdx.x; i < nkb * 32; i += kGatThreads) {
            const int k = kb0 * 32 + i;
            int2 e = make_int2(0, 0);
            if (k < a.K) {
                const int major = quotient(g.channel_last ? p.channels : p.taps, k), minor = k - major * (int)(g.channel_last ? p.channels.d : p.taps.d);
                const int c = g.channel_last ? minor : major, rs = g.channel_last ? major : minor;
                const int r = quotient(p.tap_cols, rs), s = rs - r * g.S;
                e = make_int2(((c * g.H + r * g.tap_h) * g.W + s * g.tap_w) * g.N, (int)(1u << rs));
            }
            tab[i] = e;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = (unsigned)warp_uniform((int)tmem_holder);
    const unsigned tmem_sums = tmem_base + SLOTS * 64;

    if (wid >= 16 && wid < 24) {
        // ---- copies of A: a warp has eight columns of a k-block, a lane four rows of them
        constexpr int COLUMNS = 32 / (8 / COPY_GROUPS);
        constexpr int ROWS = WIDE ? 1 : 4;                       // bases of a lane
        const int cg = (wid - 16) / (8 / COPY_GROUPS), first = (wid & (8 / COPY_GROUPS - 1)) * COLUMNS;
        const float* base[ROWS];
        unsigned mask[ROWS];                                     // bit t: tap t inside
#pragma unroll
        for (int e = 0; e < ROWS; ++e) {
            const int row = m0 + (WIDE ? lane * 4 : lane + 32 * e);
            mask[e] = 0;
            base[e] = (const float*)a.A;
            if (row < a.M) {
                const int pq = quotient(p.images, row), n = row - pq * g.N, pp = quotient(p.cols, pq), q = pq - pp * g.Q;
                const int h0 = pp * g.step_h + g.off_h, w0 = q * g.step_w + g.off_w;
                for (int r = 0, t = 0; r < g.R; ++r)
                    for (int s = 0; s < g.S; ++s, ++t) {
                        const int hh = h0 + r * g.tap_h, ww = w0 + s * g.tap_w;
                        if (hh >= 0 && hh < g.H && ww >= 0 && ww < g.W) mask[e] |= 1u << t;
                    }
                base[e] += ((long long)h0 * g.W + w0) * g.N + n;
            }
        }
        asm volatile("griddepcontrol.wait;" ::: "memory");
        bool ok = true;
        int s = cg % NR;
        unsigned bits = 0;                                       // (bit s: parity of the next phase of stage s)
        for (int kb = cg; kb < nkb; kb += COPY_GROUPS) {
            if (ok && kb >= NR) {
                if (!mbar_wait(&raw_empty[cg][s], (bits >> s) & 1u)) { atomicExch(&fail_flag, 1); ok = false; }
                bits ^= 1u << s;
            }
            const int4* t = (const int4*)(tab + kb * 32 + first);        // two columns to a load
            const unsigned to = smem_u32(ring + s * kGatRaw) + first * kGatLine + (WIDE ? lane * 16 : lane * 4);
#pragma unroll
            for (int i = 0; i < COLUMNS; i += 2) {
                const int4 e = t[i >> 1];
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    // (no byte is read where the tap lies outside)
                    if (WIDE) {
                        cp_async16(to + i * kGatLine, base[r] + e.x, mask[r] & (unsigned)e.y ? 16 : 0);
                        cp_async16(to + (i + 1) * kGatLine, base[r] + e.z, mask[r] & (unsigned)e.w ? 16 : 0);
                    } else {
                        cp_async4(to + i * kGatLine + r * 128, base[r] + e.x, mask[r] & (unsigned)e.y ? 4 : 0);
                        cp_async4(to + (i + 1) * kGatLine + r * 128, base[r] + e.z, mask[r] & (unsigned)e.w ? 4 : 0);
                    }
                }
            }
            cp_async_arrive(&raw_full[kb % GROUPS][s]);
            s += COPY_GROUPS;
            if (s >= NR) s -= NR;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (wid < 16) {
        // ---- converters
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (threadIdx.x < BN) {
            const int col = n0 + (int)threadIdx.x;
            bias[threadIdx.x] = a.bias && col < a.N ? __ldg(a.bias + (a.b_kind == B2_OPERAND_FILTER ? col - quotient(p.pixel, col) * g.kt : col)) : 0.0f;
        }
        const int group = wid >> 3, quarter = wid & 3, half = wid >> 2 & 1, row = quarter * 32 + lane;
        bool ok = true;
        int s = group % NR, slot = group % SLOTS;
        unsigned raw_bits = 0;
        for (int kb = group; kb < nkb; kb += GROUPS) {
            const unsigned slot_a = tmem_base + slot * 64 + half * 16 + ((unsigned)(quarter * 32) << 16);
            if (ok && !mbar_wait(&raw_full[group][s], (raw_bits >> s) & 1u)) { atomicExch(&fail_flag, 1); ok = false; }
            raw_bits ^= 1u << s;
            unsigned v[16], hi[16], lo[16];
            raw_row<MODE, 128, B2_OPERAND_ROWS, 16>(ring + s * kGatRaw, row, half * 16, 0, 0, v);
            to_planes<MODE, 16>(v, hi, lo);
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_empty[(kb + NR) % COPY_GROUPS][s]);
            if (kb >= SLOTS) {
                if (ok && !mbar_wait(&slot_empty[slot], (kb / SLOTS - 1) & 1)) { atomicExch(&fail_flag, 1); ok = false; }
                tc_fence_after();
            }
            tmem_st<16>(slot_a, hi);
            tmem_st<16>(slot_a + 32, lo);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&slot_full[slot]);
            s += GROUPS;
            if (s >= NR) s -= NR;
            slot += GROUPS;
            if (slot >= SLOTS) slot -= SLOTS;
        }
    } else if (wid == 25) {
        if (elect_one()) {
            // ---- copies of B: one to a k-block, in the order of n tiles and k-blocks
            asm volatile("griddepcontrol.wait;" ::: "memory");
            const char* src = (const char*)a.staged + ((long long)blockIdx.x * p.num_kb + kb0) * PLANES;
            int s = 0, n = 0;
            unsigned parity = 1;
            for (; n < nkb; ++n) {
                if (!mbar_wait(&b_empty[s], parity)) { atomicExch(&fail_flag, 1); break; }
                mbar_expect_tx(&b_full[s], PLANES);
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                    ::"r"(smem_u32(planes + s * PLANES)), "l"(src + (long long)n * PLANES), "r"(PLANES),
                      "r"(smem_u32(&b_full[s])) : "memory");
                if (++s == NB) { s = 0; parity ^= 1u; }
            }
            // what is in flight lands before the block ends, whatever has become of the other roles
            for (int i = n > NB ? n - NB : 0; i < n; ++i)
                if (!mbar_wait(&b_full[i % NB], (i / NB) & 1)) { atomicExch(&fail_flag, 1); break; }
        }
    } else if (wid == 24 || ISSUERS > 1) {
        if (elect_one()) {
            // ---- MMA issue.  K-block n of K (not of the slice: the planes' order goes by it) is issuer n % ISSUERS's, and
            // its hh n / ISSUERS % 2.
            const unsigned id1 = make_idesc(1, 2, 2, BN), id2 = make_idesc(1, 2, 2, 2 * BN);
            const unsigned long long desc = make_smem_desc(planes);
            const int mine = wid == 24 ? 0 : 1;
            const unsigned base = tmem_sums + mine * gat_group(BN), x = base + BN;
            unsigned begun = 0;                                   // bit h: hh h has a k-block
            int kb = (kb0 + mine) % ISSUERS;
            for (; kb < nkb; kb += ISSUERS) {
                const int slot = kb % SLOTS, b = kb % NB;
                if (!mbar_wait(&b_full[b], (kb / NB) & 1) || !mbar_wait(&slot_full[slot], (kb / SLOTS) & 1)) { atomicExch(&fail_flag, 1); break; }
                tc_fence_after();
                const unsigned ah = tmem_base + slot * 64, al = ah + 32;
                const bool turned = (kb0 + kb) / ISSUERS & 1;        // [lo | hi]
                const unsigned hh = turned ? x + BN : base, both = turned ? x : base;
                const unsigned long long d0 = desc + (unsigned)(b * PLANES >> 4);
                const unsigned long long dH = turned ? d0 + (BN * 128 >> 4) : d0, dL = turned ? d0 : d0 + (BN * 128 >> 4);
                const bool fresh = !(begun >> turned & 1u);
                if (fresh && begun) {                             // a new hh beside an x with sums in it
                    tc_mma_ta<MODE>(hh, ah, dH, id1, 0u);
                    tc_mma_ta<MODE>(x, ah, dL, id1, 1u);
                } else {
                    tc_mma_ta<MODE>(both, ah, d0, id2, fresh ? 0u : 1u);
                }
                tc_mma_ta<MODE>(x, al, dH, id1, 1u);
#pragma unroll
                for (int k = 1; k < 4; ++k) {
                    tc_mma_ta<MODE>(both, ah + 8 * k, d0 + 2 * k, id2, 1u);
                    tc_mma_ta<MODE>(x, al + 8 * k, dH + 2 * k, id1, 1u);
                }
                tc_commit(&slot_empty[slot]);
                tc_commit(&b_empty[b]);
                begun |= 1u << turned;
            }
            tc_commit(&sums_full);
        }
    }
    __syncwarp();

    // ---- epilogue: the sixteen converting warps; lane quarter = warp % 4, the four warps of a quarter take the
    // 8-column pieces in turn
    float* red = (float*)smem;                                    // [BN][128], slices only
    const int quarter = wid & 3, part = wid >> 2, lrow = quarter * 32 + lane, row = m0 + lrow;
    const int splits = p.splits;
    const bool tiled = a.b_kind == B2_OPERAND_FILTER;
    // tiles of several pixels: where the row's tile starts
    int tile_p = 0, tile_q = 0;
    long long tile_at = row;
    if (tiled) {
        const int pq = quotient(p.images, row), n = row - pq * g.N, pp = quotient(p.cols, pq);
        tile_p = pp * g.gh; tile_q = (pq - pp * g.Q) * g.gw;
        tile_at = ((long long)tile_p * g.out_q + tile_q) * g.N + n;
    }
    // a thread's columns: groups of eight, or of four where slices are exchanged.  Where the first of one goes, and how
    // many of it exist
    const int start = splits == 1 ? part * 8 : (rank + part * splits) * 4, stride = splits == 1 ? 32 : 16 * splits;
    auto group_at = [&](int c0, long long& at) -> int {
        int col = n0 + c0;
        const int live = a.N - col;
        at = tile_at;
        if (row >= a.M || live <= 0) return 0;
        if (tiled) {
            const int pix = quotient(p.pixel, col), gy = quotient(p.pixel_cols, pix), gx = pix - gy * g.gw;
            col -= pix * g.kt;
            if (tile_p + gy >= g.out_p || tile_q + gx >= g.out_q) return 0;
            at += ((long long)gy * g.out_q + gx) * g.N;
        }
        at += (long long)col * a.ldc;
        return live;
    };
    // Residual and mask of a group, the next one's under way while one is finished.  Choices are made once a group: with
    // a branch for each of a value's terms eight values took 1600 cycles.
    constexpr int OWN = (BN + 31) / 32;                           // groups of a thread
    float residual[8], mask[8];
    auto fetch = [&](int c0, auto w) {
        constexpr int W = decltype(w)::value;
        long long at;
        const int live = c0 < BN ? group_at(c0, at) : 0;
        auto eight = [&](const float* from, float* to) {
            if (live >= W) {
#pragma unroll
                for (int j = 0; j < W; ++j, from += a.ldc) to[j] = __ldg(from);
            } else {
#pragma unroll
                for (int j = 0; j < W; ++j) to[j] = j < live ? __ldg(from + j * a.ldc) : 0.0f;
            }
        };
        if (a.residual) eight(a.residual + at, residual);
        if (a.mask) eight(a.mask + at, mask);
    };
    // the group of the columns from c0 on: tail and store; then the next one's terms
    auto finish = [&](int c0, auto w, float* y) {
        constexpr int W = decltype(w)::value;
        long long at;
        const int live = group_at(c0, at);
        if (a.bias) {
#pragma unroll
            for (int j = 0; j < W; ++j) y[j] += bias[c0 + j];
        }
        if (a.residual) {
#pragma unroll
            for (int j = 0; j < W; ++j) y[j] += residual[j];
        }
        if (a.relu) {
#pragma unroll
            for (int j = 0; j < W; ++j) y[j] = y[j] < 0.0f ? 0.0f : y[j];      // (keeps NaN, as max(x, 0) does)
        }
        if (a.mask) {
#pragma unroll
            for (int j = 0; j < W; ++j) y[j] *= mask[j] > 0.0f ? 1.0f : 0.0f;     // (likewise)
        }
        if (a.residual || a.mask) fetch(c0 + stride, w);
        float* out = (float*)a.C + at;
        if (live >= W) {
#pragma unroll
            for (int j = 0; j < W; ++j, out += a.ldc) *out = y[j];
        } else {
#pragma unroll
            for (int j = 0; j < W; ++j)
                if (j < live) out[j * a.ldc] = y[j];
        }
    };
    if (wid < 16 && (a.residual || a.mask)) {
        if (splits == 1) fetch(start, std::integral_constant<int, 8>());
        else fetch(start, std::integral_constant<int, 4>());
    }
    bool ok = true;
    if (wid < 16) {
        ok = mbar_wait(&sums_full, 0);
        if (!ok) atomicExch(&fail_flag, 1);
        asm volatile("bar.sync 1, 512;" ::: "memory");            // (the biases)
        tc_fence_after();
        const unsigned lane_addr = tmem_sums + ((unsigned)(quarter * 32) << 16);
#pragma unroll 1
        for (int i = 0; i < OWN; ++i) {
            const int c0 = part * 8 + 32 * i;
            if (c0 >= BN || n0 + c0 >= a.N) break;
            // the sums that there are: all hh, all x
            float hh[8], xx[8];
            unsigned h[8], x[8];
#pragma unroll
            for (int q = 0; q < ISSUERS; ++q) {
                const int issuer = (kb0 + q) % ISSUERS;           // k-blocks q, q + ISSUERS, ... of the slice
                if (q >= nkb) break;
                const unsigned at = lane_addr + issuer * gat_group(BN) + c0;
                const unsigned head = (unsigned)((kb0 + q) / ISSUERS & 1) * 2 * BN;
                const bool second = q + ISSUERS < nkb;
                unsigned h2[8];
                tmem_ld8(at + head, h);
                tmem_ld8(at + BN, x);
                if (second) tmem_ld8(at + 2 * BN - head, h2);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    hh[j] = q ? hh[j] + __uint_as_float(h[j]) : __uint_as_float(h[j]);
                    xx[j] = q ? xx[j] + __uint_as_float(x[j]) : __uint_as_float(x[j]);
                }
                if (second) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) hh[j] += __uint_as_float(h2[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) hh[j] += xx[j];
            if (splits == 1) {
                if (ok) finish(c0, std::integral_constant<int, 8>(), hh);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) red[(c0 + j) * 128 + lrow] = hh[j];
            }
        }
    }
    if (splits > 1) {
        cluster_sync();
        if (wid < 16) {
            // this CTA's share of the columns: groups of four, every splits-th, dealt to the warps of a quarter
#pragma unroll 1
            for (int i = 0; i < OWN; ++i) {
                const int c0 = start + i * stride;
                if (c0 >= BN) break;
                if (n0 + c0 >= a.N) break;
                float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                // (a peer's values take about 700 cycles: those of several slices come together)
                constexpr int Z = 4;
                for (int z0 = 0; z0 < splits; z0 += Z) {
                    float t[Z][4];
#pragma unroll
                    for (int z = 0; z < Z; ++z) {
                        if (z0 + z >= splits) break;
                        const unsigned at = map_rank(red + c0 * 128 + lrow, z0 + z);
#pragma unroll
                        for (int j = 0; j < 4; ++j) t[z][j] = ld_peer(at + j * 512, 0.0f);
                    }
#pragma unroll
                    for (int z = 0; z < Z; ++z) {
                        if (z0 + z >= splits) break;
#pragma unroll
                        for (int j = 0; j < 4; ++j) v[j] += t[z][j];
                    }
                }
                if (ok) finish(c0, std::integral_constant<int, 4>(), v);
            }
        }
        cluster_sync();                                           // peers may still be reading
    }
    tc_fence_before();
    __syncthreads();
    if (wid == 24) {
        tc_fence_after();
        tmem_dealloc(tmem_base, gat_tmem(BN));
    }
    if (threadIdx.x == 0 && fail_flag && a.status) atomicExch(a.status, 1);
}

// ---- host ------------------------------------------------------------------------------------
struct GatherShape { int bn, splits, kb_per_split, waves; long long cost; };

int gather_smem(int bn, int kb_per_split) {
    int smem = gat_b_stages(bn) * 2 * bn * 128 + kGatRawStages * kGatRaw + kb_per_split * 32 * 8;
    if (bn * 128 * 4 > smem) smem = bn * 128 * 4;
    return smem + 1024;
}

GatherShape gather_shape(const b2_direct_args& a) {
    const int num_kb = (a.K + 31) / 32;
    GatherShape best = {0, 0, 0, 0, -1};
    const long long tm = (a.M + 127) / 128;
    if (tm > 65535) return best;
    int per_of[9] = {};                                           // k-blocks of a slice, 0: not so many slices
    for (int want = 1; want <= 8 && want <= num_kb; ++want) {
        const int per = (num_kb + want - 1) / want;
        if ((want - 1) * per < num_kb) per_of[want] = per;
    }
    for (int bn : {16, 32, 64, 96, 128}) {
        if (bn > 16 && (bn == 96 ? 64 : bn / 2) >= a.N) break;
        const long long tiles = tm * ((a.N + bn - 1) / bn);
        const int kb = bn <= 64 ? 520 : 6 * bn + 30;
        for (int splits = 1; splits <= 8; ++splits) {
            const int per = per_of[splits];
            if (!per || gather_smem(bn, per) > 232448 - 1024) continue;
            if (a.longest > 0 && (per + gat_sums(bn) - 1) / gat_sums(bn) > a.longest) continue;
            const long long one = 7500 + per * kb + 30 * bn + (splits == 1 ? 0 : 3000 + 10 * bn);
            if (best.cost >= 0 && one >= best.cost) continue;
            const long long ctas = tiles * splits, slots = kClusterCtas[splits], waves = (ctas + slots - 1) / slots;
            if (best.cost < 0 || waves * one < best.cost) best = {bn, splits, per, (int)waves, waves * one};
        }
    }
    return best;
}

template <int BN, bool WIDE>
int gather_launch_as(const GatherParams& p, cudaStream_t st) {
    static_assert(gat_slots(BN) * 64 + gat_issuers(BN) * gat_group(BN) <= 512, "tensor memory");
    static bool attr_set = false;
    if (!attr_set) {
        B2_CUDA(cudaFuncSetAttribute(gather_kernel<BN, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448 - 1024));
        attr_set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.a.N + BN - 1) / BN, (p.a.M + 127) / 128, p.splits);
    cfg.blockDim = dim3(kGatThreads);
    cfg.dynamicSmemBytes = gather_smem(BN, p.kb_per_split);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = p.splits;
    cfg.attrs = attr;
    cfg.numAttrs = p.splits > 1 ? 2 : 1;
    B2_CUDA(cudaLaunchKernelEx(&cfg, gather_kernel<BN, WIDE>, p));
    return B2_OK;
}

template <int BN>
int gather_launch_bn(const GatherParams& p, cudaStream_t st) {
    return ((uintptr_t)p.a.A & 15) == 0 ? gather_launch_as<BN, true>(p, st) : gather_launch_as<BN, false>(p, st);
}

}  // namespace

// Images of a pixel in fours: sixteen bytes a copy.
bool b2_gather_streams(const b2_direct_args& a) {
    return a.staged && !a.staged_own && !a.flex && a.a_kind == B2_OPERAND_GATHER && a.colmajor && a.g.N % 4 == 0;
}

b2_gather_info b2_gather_plan(const b2_direct_args& a) {
    const GatherShape s = gather_shape(a);
    const int sums = gat_sums(s.bn), issuers = gat_issuers(s.bn);
    return {s.cost, s.bn, s.splits, s.waves, s.kb_per_split, sums, (s.kb_per_split + sums - 1) / sums,
            (s.kb_per_split + issuers - 1) / issuers, issuers};
}

int b2_gather_launch(const b2_direct_args& a, cudaStream_t st) {
    const GatherShape s = gather_shape(a);
    B2_REQUIRE(s.cost >= 0 && ((uintptr_t)a.staged & 127) == 0 && ((uintptr_t)a.A & 3) == 0, "problem outside the kernel's range");
    GatherParams p;
    p.a = a;
    p.num_kb = (a.K + 31) / 32;
    p.kb_per_split = s.kb_per_split;
    p.splits = s.splits;
    const b2_gather& g = a.g;
    p.taps = divisor(g.R * g.S); p.tap_cols = divisor(g.S); p.channels = divisor(g.channels); p.images = divisor(g.N);
    p.cols = divisor(g.Q); p.pixel = divisor(g.kt > 0 ? g.kt : 1); p.pixel_cols = divisor(g.gw > 0 ? g.gw : 1);
    switch (s.bn) {
        case 16: return gather_launch_bn<16>(p, st);
        case 32: return gather_launch_bn<32>(p, st);
        case 64: return gather_launch_bn<64>(p, st);
        case 96: return gather_launch_bn<96>(p, st);
        default: return gather_launch_bn<128>(p, st);
    }
}
