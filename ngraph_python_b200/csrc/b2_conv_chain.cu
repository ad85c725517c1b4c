// A run of flex16 convolution layers in ONE launch: every CTA carries one or two images through all of
// them, with the activations between the layers in shared memory.
//
// Layer by layer (b2_conv.cu) a convolution of a small network is a launch of 5 to 15 us in which every
// CTA starts up, reads its operands from L2, and stores what the next launch reads again; ResNet-20 has
// 22 of them.  Its images do not depend on one another, and the activations of one (16 channels of 32x32:
// 36 KB as two byte planes) fit into an SM three times over.  So a CTA keeps them there, and per layer only
// the filters come in (one bulk copy, while the layer before is at work).
//
// Operands.  In shared memory a tensor is [high, low byte plane][groups of 16 channels][row][image][column]
// of 16 bytes -- the 16 channels of a pixel -- with a ring of zero pixels around every image.  That is a
// K-major operand without swizzle: 8 neighbouring pixels are a core matrix (8 rows x 16 bytes), and the
// pixels under a tap of the filter are the same pixels at another start address, so nothing is unrolled.
// An MMA's 128 rows are 16 groups of 8 neighbouring columns, a row of an image each; its 32 bytes of K are
// two (tap, channel group) chunks, whose distance is the descriptor's leading byte offset.  With two images
// their rows alternate, which keeps the distance of the groups constant across images.  A tensor that
// convolutions of stride 2 read is kept as its four parities of (row, column), so that there too
// neighbouring results read neighbouring pixels.
//
// The products are those of the tile kernel (high and low bytes, the filters' low byte stored minus 128,
// its bias undone with the sum of the activations under the window), as two instructions per k-step:
//     A_hi x [B_hi | B_lo' | sum] -> HH | X1 | S_hi        A_lo x [B_hi | B_lo' | sum] -> X2 | LL | S_lo
// (B_hi and B_lo' by turns, eight output channels each),
// each issued by a thread of its own (an MMA this small costs its issuer about as long as the tensor
// pipe).  The epilogue evaluates the layer's tail with the arithmetic of the tile kernel, operation for
// operation, so a network gives the same bits either way.  A thread has a pixel and 16 of its channels:
// what it stores is two 16-byte vectors, where the tile kernel has to turn images around.
//
// Order.  A layer's tiles follow those of the layer before as soon as the tiles around them are stored
// (`coarse` layers, which read something else or take over other memory, wait for all of them).  The
// single pass over tiles is what makes taking over the memory of tensors that are no longer read safe;
// plan() has the conditions.
//
// What bounds it: 256 images of ResNet-20 (128 CTAs of two images), 22 layers: 204 us one by one, 120 us
// here.  Of these 60 are the chain of hand-overs (issue, full set, stored tile: 2.4 us a layer), 15 the
// products beyond the first k-step of a tile, 13 the arithmetic of the epilogue and 34 the rest of it
// (operands, tails, stores); a rolled epilogue is faster than an unrolled one (120 / 135 us), because a
// warp that comes to a line of instructions after the others of its scheduler fetches it anew.
#include <algorithm>
#include <vector>

#include "b2_gemm_impl.cuh"

namespace {

constexpr int kLayersMost = B2_CONV_CHAIN_MAX;
constexpr int kStepsMost = 36;               // k-steps of 32 bytes a layer may have
constexpr int kTilesMost = 32;
constexpr int kChannelsMost = 112;           // output channels: 2 * 112 + 16 columns an accumulator
constexpr int kCtaThreads = 640;             // sixteen epilogue warps, one for the copies, three issuers
constexpr int kEpiWarps = 16;
constexpr int kSmemMost = 232448;
constexpr int kFixedUnits = 82;              // barriers, counters, biases, scales; see the kernel (16-byte units)

// A tensor in shared memory; 16-byte units throughout
struct Place {
    int off[4];                              // pixel (0, 0) of the first image (per parity of row, column)
    int pitch, grp, plane;                   // row, 16 channels, low plane behind the high one
    int parity;
};

struct Layer {
    unsigned step[kStepsMost + 1];           // operand offset of a k-step | distance of its halves << 16
    int nk, a_base, a_row, sbo, plane;
    int trows, tcols, tiles;
    int filt, filt_units, prefetch;
    long long filt_src;
    int n2, nsets, K, P, Q;
    int coarse, zero, zero_at, zero_units;
    int has_out, has_res;
    Place out, res;
    int slot_in, slot_f, slot_out, slot_bias, slot_res;
    int relu, short_sum;
    const short* bias;
    short* dst;
};

struct Chain {
    int n, N, glog;
    int inC, inH, inW;
    Place in;
    const unsigned char *src_hi, *src_lo;    // byte (c, h, w, n) at ((c*H + h)*W + w)*pitch + n*estep
    long long src_pitch;
    int src_estep;
    const unsigned char* filters;
    const b2_flex_scale* table;
    int* stats;
    int* status;
    int smem_units;
    short* pooled;                           // K x N averages of the last layer's images, or null
    Layer layer[kLayersMost];
};

__device__ __forceinline__ int pixel_at(const Place& t, int glog, int h, int img, int w) {
    const int g = t.parity ? (h & 1) * 2 + (w & 1) : 0, s = t.parity;
    return t.off[g] + (((h >> s) << glog) + img) * t.pitch + (w >> s);
}
// How far the layers have come, in counters that only grow (the phases of a barrier would have to be met
// by everyone in turn).  `done`: a word per epilogue warp, the tiles it has stored -- a sum over a set's
// warps would not tell one that is a tile ahead from one that is behind.  `drained`: a word per accumulator
// set, its warps' shares of sixteen a tile; no warp drains a tile before all have drained the one before.
__device__ __forceinline__ void count_up(unsigned* word, unsigned n) {
    asm volatile("red.release.cta.shared::cta.add.u32 [%0], %1;" ::"r"(smem_u32(word)), "r"(n) : "memory");
}
__device__ __forceinline__ void publish(unsigned* word, unsigned n) {
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(word)), "r"(n) : "memory");
}
__device__ __forceinline__ int least4(const unsigned* words) {
    int a, b, c, d;
    asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(smem_u32(words)) : "memory");
    return min(min(a, b), min(c, d));
}
// waits until the four warps of every slot have stored at least so many tiles; for ONE thread of a warp
__device__ __forceinline__ bool stored(const unsigned* done, int4 e, unsigned pause = 20) {
    for (int i = 0; i < kWaitPolls; ++i) {
        const int a = least4(done) - e.x, b = least4(done + 4) - e.y, c = least4(done + 8) - e.z, d = least4(done + 12) - e.w;
        if (min(min(a, b), min(c, d)) >= 0) {
            asm volatile("fence.acq_rel.cta;" ::: "memory");
            return true;
        }
        if (pause) __nanosleep(pause);           // (polling takes issue slots from the epilogue warps)
    }
    return false;
}
__device__ __forceinline__ bool counted(const unsigned* word, unsigned e) {
    for (int i = 0; i < kWaitPolls; ++i) {
        unsigned v;
        asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(word)) : "memory");
        if ((int)(v - e) >= 0) return true;
        __nanosleep(20);
    }
    return false;
}
// Tiles of the four slots of warps after the first n of a layer with nsets accumulator sets (a set's warps
// are 4 / nsets slots)
__device__ __forceinline__ int4 slots_after(int4 v, int n, int nsets) {
    if (nsets == 4) { v.x += (n + 3) >> 2; v.y += (n + 2) >> 2; v.z += (n + 1) >> 2; v.w += n >> 2; }
    else if (nsets == 2) { v.x += (n + 1) >> 1; v.y += (n + 1) >> 1; v.z += n >> 1; v.w += n >> 1; }
    else { v.x += n; v.y += n; v.z += n; v.w += n; }
    return v;
}
// uses of the accumulator sets
__device__ __forceinline__ int4 sets_after(int4 v, int n, int nsets) {
    if (nsets == 4) return slots_after(v, n, 4);
    if (nsets == 2) { v.x += (n + 1) >> 1; v.y += n >> 1; }
    else v.x += n;
    return v;
}
// A bounded wait that suspends for up to 0.1 ms at a time: many warps wait here, and a poll takes issue slots
// from those that work.
__device__ __forceinline__ bool bar_wait(unsigned long long* bar, unsigned parity) {
    for (int i = 0; i < 1024; ++i) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(100000) : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void epilogue_barrier() {
    asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
}
__device__ __forceinline__ unsigned tmem_ld1(unsigned taddr) {
    unsigned r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(taddr) : "memory");
    return r;
}

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Eight columns of an accumulator set (v1: HH | X1, v2: X2 | LL) to four pairs of mantissas.  The arithmetic
// of conv_implicit_kernel's fused epilogue: same operations, same order; what differs is how the result is
// quantised (rounded to nearest even and saturated by the conversions, the same values).
template <bool SHORT>
__device__ __forceinline__ void finish8(const unsigned* v1, const unsigned* v2, unsigned long long fix,
                                        unsigned long long f, const unsigned long long* y, unsigned* w) {
    const unsigned long long k256 = pack2(256.0f, 256.0f), k65536 = pack2(65536.0f, 65536.0f);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        const unsigned xa = v1[8 + j] + v2[j], xb = v1[9 + j] + v2[j + 1];
        const unsigned long long l = add2(pack2((float)(int)v2[8 + j], (float)(int)v2[9 + j]), fix);
        unsigned long long v;
        if (SHORT)
            v = fma2(pack2((float)(int)((v1[j] << 8) + xa), (float)(int)((v1[j + 1] << 8) + xb)), k256, l);
        else
            v = fma2(pack2((float)(int)v1[j], (float)(int)v1[j + 1]), k65536, fma2(pack2((float)(int)xa, (float)(int)xb), k256, l));
        v = fma2(v, f, y[j >> 1]);
        float p, q;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(p), "=f"(q) : "l"(v));
        asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(w[j >> 1]) : "r"(__float2int_rn(q)), "r"(__float2int_rn(p)));
    }
}

// Eight channels of a pixel into an int16 tensor (results that somebody outside the chain reads; a call, so
// that the loop around it stays short)
__device__ __noinline__ void store8(short* o, long long step, unsigned a, unsigned b, unsigned c, unsigned d) {
    o[0] = (short)a; o[step] = (short)(a >> 16);
    o[2 * step] = (short)b; o[3 * step] = (short)(b >> 16);
    o[4 * step] = (short)c; o[5 * step] = (short)(c >> 16);
    o[6 * step] = (short)d; o[7 * step] = (short)(d >> 16);
}

__global__ void __launch_bounds__(kCtaThreads, 1)
conv_chain_kernel(const __grid_constant__ Chain p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    // fixed part: barriers, then the biases of two layers, then the layers' scales
    unsigned char* fixed = smem + (size_t)p.smem_units * 16;
    unsigned long long* filt_full = (unsigned long long*)fixed;            // [2]
    unsigned long long* tmem_full = filt_full + 2;                         // [4]
    unsigned* drained = (unsigned*)(tmem_full + 4);                        // [4] accumulator sets read
    unsigned* done = drained + 4;                                          // [4 slots][4 quarters] tiles stored
    unsigned long long* issued = (unsigned long long*)(done + 16);         // the last instructions have run
    unsigned* tmem_holder = (unsigned*)(issued + 1);
    int* fail_flag = (int*)(tmem_holder + 1);
    float* bias_s = (float*)(fixed + 144);                                 // [2][kChannelsMost]
    float2* scale_s = (float2*)(fixed + 144 + 2 * kChannelsMost * 4);      // [kLayersMost] (conv, residual)

    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int glog = p.glog, G = 1 << glog, n0 = (int)blockIdx.x << glog;
    const int n_img = p.N - n0 < G ? p.N - n0 : G;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) mbar_init(&filt_full[i], 1);
        // (a tile's instructions come from one thread or from two: two arrivals)
        for (int i = 0; i < 4; ++i) { mbar_init(&tmem_full[i], 2); drained[i] = 0; }
        for (int i = 0; i < 16; ++i) done[i] = 0;
        mbar_init(issued, 3);
        *fail_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kEpiWarps + 1) {
        tmem_alloc(tmem_holder, 512);
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    // the rings of zero pixels (and everything else: tensors that come later rely on it)
    for (int i = threadIdx.x; i < p.smem_units; i += kCtaThreads)
        reinterpret_cast<uint4*>(smem)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (threadIdx.x < p.n) {
        const Layer& L = p.layer[threadIdx.x];
        const float q = p.table[L.slot_out].inv_scale;
        scale_s[threadIdx.x] = make_float2(p.table[L.slot_in].scale * p.table[L.slot_f].scale * q,
                                           L.has_res ? p.table[L.slot_res].scale * q : 0.0f);
    }
    // the images: a thread has four pixels and 16 channels, four of them at a time (neighbouring pixels lie
    // N images apart: a load brings 32 lines, so all that a thread has are in flight together)
    {
        const int pixels = p.inH * p.inW << glog, units = pixels * ((p.inC + 15) >> 4);
        const long long cs = (long long)p.inH * p.inW * p.src_pitch;
        for (int i0 = threadIdx.x; i0 < units; i0 += 4 * kCtaThreads) {
            int at[4], c0[4];
            long long from[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = i0 + j * kCtaThreads, g = i / pixels, r = i - g * pixels;
                const int img = r & (G - 1), hw = r >> glog, h = hw / p.inW, w = hw - h * p.inW;
                const bool there = i < units && img < n_img;
                at[j] = there ? pixel_at(p.in, glog, h, img, w) + g * p.in.grp : -1;
                c0[j] = there ? g * 16 : p.inC;
                from[j] = g * 16 * cs + hw * p.src_pitch + (long long)(n0 + img) * p.src_estep;
            }
            unsigned hi[4][4], lo[4][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (q * 4 >= p.inC) {                          // (fewer than 16 channels in all)
#pragma unroll
                    for (int j = 0; j < 4; ++j) hi[j][q] = lo[j][q] = 0;
                    continue;
                }
                unsigned v[4][4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const long long o = from[j] + (q * 4 + k) * cs;
                        v[j][k] = 0;
                        if (c0[j] + q * 4 + k < p.inC)
                            v[j][k] = p.src_estep == 2 ? *reinterpret_cast<const unsigned short*>(p.src_lo + o)
                                                       : (unsigned)p.src_hi[o] << 8 | p.src_lo[o];
                    }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const unsigned a = v[j][0] | v[j][1] << 16, b = v[j][2] | v[j][3] << 16;
                    lo[j][q] = __byte_perm(a, b, 0x6420);
                    hi[j][q] = __byte_perm(a, b, 0x7531);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (at[j] >= 0) {
                    uint4* d = reinterpret_cast<uint4*>(smem) + at[j];
                    d[0] = make_uint4(hi[j][0], hi[j][1], hi[j][2], hi[j][3]);
                    d[p.in.plane] = make_uint4(lo[j][0], lo[j][1], lo[j][2], lo[j][3]);
                }
        }
    }
    fence_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = (unsigned)warp_uniform((int)*tmem_holder);

    if (warp == kEpiWarps) {
        // filters and biases of layer l, while layer l-1 is at work where the memory for them is free then
        // (prefetch), else once it is done
        int finished = 0, l = 0;                // layers whose every tile is stored
        int4 e = make_int4(0, 0, 0, 0);
        bool ok = true;
        for (; l < p.n; ++l) {
            const Layer& L = p.layer[l];
            for (const int need = l - (L.prefetch ? 1 : 0); finished < need; ++finished)
                e = slots_after(e, p.layer[finished].tiles, p.layer[finished].nsets);
            // One lane looks.  (A 16-byte load of the whole warp is two passes, and what lies there may change
            // between them: half the lanes would go on without the other half, whatever the compiler takes
            // a load from one address to be.)
            int go = 1;
            if (lane == 0) go = stored(done, e, 200);
            ok = __shfl_sync(0xffffffffu, go, 0) != 0;
            if (!ok) break;
            float* b = bias_s + (l & 1) * kChannelsMost;
            for (int k = lane; k < L.K; k += 32)
                b[k] = L.bias ? (float)L.bias[k] * p.table[L.slot_bias].scale * p.table[L.slot_out].inv_scale : 0.0f;
            __syncwarp();
            if (lane == 0) {
                fence_async();
                mbar_expect_tx(&filt_full[l & 1], L.filt_units * 16);
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                    ::"r"(smem_u32(smem) + L.filt * 16), "l"(p.filters + L.filt_src), "r"(L.filt_units * 16),
                      "r"(smem_u32(&filt_full[l & 1])) : "memory");
            }
            __syncwarp();
        }
        // what is in flight lands before the block ends, whatever has become of the other roles
        if (lane == 0) {
            for (int i = l > 2 ? l - 2 : 0; i < l; ++i)
                if (!bar_wait(&filt_full[i & 1], (i >> 1) & 1u)) ok = false;
            if (!ok) atomicExch(fail_flag, 1);
        }
        __syncwarp();
    } else if (warp > kEpiWarps) {
        // The issuing threads take a layer's tiles in turn; where there is one tile only, the first two
        // share it, one the high bytes of the activations, one the low ones.  (Each is a chain of waits
        // and instructions; three of them keep the sixteen warps behind them busy.)
        const int mine = warp - kEpiWarps - 1;
        if (elect_one()) {
            const unsigned smem_lo = smem_u32(smem) >> 4;
            const unsigned id_hi = make_idesc(2, 1, 1, 0), id_lo = make_idesc(2, 0, 1, 0);
            int4 prev = make_int4(0, 0, 0, 0), base = prev, uses = prev;     // tiles before the last layer, before this one
            int prev_sets = 4;
            bool ok = true;
            for (int l = 0; l < p.n && ok; ++l) {
                const Layer& L = p.layer[l];
                const int nk = L.nk, nsets = L.nsets, n2 = L.n2, tiles = L.tiles, tcols = L.tcols;
                const bool split = tiles == 1;
                const unsigned long long a_hi = ((unsigned long long)(unsigned)L.sbo << 32) | (1ULL << 46),
                                         b_hi = ((unsigned long long)8u << 32) | (1ULL << 46);
                const unsigned b_step = 2u * n2, b_lo = (smem_lo + L.filt) | (unsigned)n2 << 16, nbits = (unsigned)(n2 >> 3) << 17;
                const int a_row = L.a_row, plane = L.plane, coarse = L.coarse;
                const unsigned a_base = smem_lo + L.a_base;
                bool first = true;
                for (int t = split ? 0 : mine; t < tiles && (!split || mine < 2); t += split ? 1 : 3) {
                    const int tr = t / tcols, tc = t - tr * tcols, s = t & (nsets - 1);
                    const unsigned d = tmem_base + (unsigned)(2 * s * n2);
                    const unsigned a0 = a_base + (unsigned)(tr * a_row + tc * 8);
                    const unsigned used = 16u * (unsigned)((s == 0 ? uses.x : s == 1 ? uses.y : s == 2 ? uses.z : uses.w) + t / nsets);
                    unsigned b = b_lo, nxt = L.step[0], acc = 0;
                    if (coarse) {
                        if (first && ok) ok = stored(done, base);
                    } else if (ok) {
                        // (the layer before has the same tiles)
                        const int er = tr + 1 < L.trows ? tr + 1 : tr, ec = tc + 1 < tcols ? tc + 1 : tc;
                        ok = stored(done, slots_after(prev, er * tcols + ec + 1, prev_sets));
                    }
                    if (first && ok) ok = bar_wait(&filt_full[l & 1], (l >> 1) & 1u);
                    first = false;
                    if (!ok || !counted(&drained[s], used)) { ok = false; break; }
                    tc_fence_after();
                    if (!split) {
                        const unsigned ih = id_hi | nbits, il = id_lo | nbits, dl = d + n2;
#pragma unroll 2
                        for (int k = 0; k < nk; ++k, b += b_step) {
                            const unsigned st = a0 + nxt;
                            nxt = L.step[k + 1];                               // (the table has one to spare)
                            tc_mma<MODE_FLEX16>(d, a_hi | st, b_hi | b, ih, acc);
                            tc_mma<MODE_FLEX16>(dl, a_hi | (st + plane), b_hi | b, il, acc);
                            acc = 1;
                        }
                    } else {
                        const unsigned id = (mine ? id_lo : id_hi) | nbits, dd = d + mine * n2, aa = a0 + mine * plane;
#pragma unroll 2
                        for (int k = 0; k < nk; ++k, b += b_step) {
                            const unsigned st = aa + nxt;
                            nxt = L.step[k + 1];
                            tc_mma<MODE_FLEX16>(dd, a_hi | st, b_hi | b, id, acc);
                            acc = 1;
                        }
                    }
                    if (!split) mbar_arrive(&tmem_full[s]);
                    tc_commit(&tmem_full[s]);
                }
                prev = base; prev_sets = nsets;
                base = slots_after(base, tiles, nsets);
                uses = sets_after(uses, tiles, nsets);
            }
            // nothing of this thread's is at work any more when the block ends, also where a wait ran out
            tc_commit(issued);
            if (!bar_wait(issued, 0)) ok = false;
            if (!ok) atomicExch(fail_flag, 1);
        }
    } else {
        const int quarter = warp & 3, slot = warp >> 2;
        // this thread's pixel in the first tile; a tile further down is 16 >> glog rows of the images
        const int row8 = quarter * 4 + (lane >> 3), h0 = row8 >> glog, img = row8 & (G - 1), q0 = lane & 7;
        unsigned full_bits = 0, stored_tiles = 0;
        bool ok = true;
        for (int l = 0; l < p.n; ++l) {
            const Layer& L = p.layer[l];
            if (L.coarse && l > 0) epilogue_barrier();          // the layer before is stored
            if (L.zero) {
                for (int i = threadIdx.x; i < L.zero_units; i += kEpiWarps * 32)
                    reinterpret_cast<uint4*>(smem)[L.zero_at + i] = make_uint4(0, 0, 0, 0);
                fence_async();
                epilogue_barrier();
            }
            const int nsets = L.nsets, epi_w = 4 / nsets, set = slot / epi_w, part = slot - set * epi_w;
            const int kt = L.K, n2 = L.n2, tiles = L.tiles, tcols = L.tcols;
            const float2 sc = scale_s[l];
            const unsigned long long f = pack2(sc.x, sc.x), r = pack2(sc.y, sc.y);
            const float* bias = bias_s + (l & 1) * kChannelsMost;
            const unsigned d1 = tmem_base + (unsigned)(2 * set * n2) + ((unsigned)(quarter * 32) << 16), d2 = d1 + n2;
            const bool has_res = L.has_res && img < n_img, has_out = L.has_out && img < n_img, short_sum = L.short_sum;
            const int P = L.P, Q = L.Q, out_grp = L.out.grp, out_plane = L.out.plane, res_grp = L.res.grp, res_plane = L.res.plane;
            const int out_at = pixel_at(L.out, glog, h0, img, q0), res_at = pixel_at(L.res, glog, h0, img, q0);
            const int out_tr = L.out.pitch * (L.out.parity ? 8 : 16), out_tc = L.out.parity ? 4 : 8;
            const int res_tr = L.res.pitch * (L.res.parity ? 8 : 16), res_tc = L.res.parity ? 4 : 8;
            const unsigned floor2 = L.relu ? 0u : 0x80008000u;
            short* const store = L.dst;
            unsigned smx = 0, smn = 0;                             // pairs: largest and smallest mantissa
            int tr = set / tcols, tc = set - tr * tcols;
            for (int t = set; t < tiles; t += nsets) {
                const int h = h0 + tr * (16 >> glog), q = q0 + tc * 8;
                const bool live = h < P && q < Q && img < n_img;
                uint4* const dst = reinterpret_cast<uint4*>(smem) + out_at + tr * out_tr + tc * out_tc;
                const uint4* const rsd = reinterpret_cast<const uint4*>(smem) + res_at + tr * res_tr + tc * res_tc;
                if (ok && !bar_wait(&tmem_full[set], full_bits >> set & 1u)) { ok = false; atomicExch(fail_flag, 1); }
                full_bits ^= 1u << set;
                tc_fence_after();
                const unsigned s_hi = tmem_ld1(d1 + 2 * kt), s_lo = tmem_ld1(d2 + 2 * kt);
                // eight channels at a time (rolled: the instructions of an unrolled tile would be fetched anew
                // by every warp that comes to them)
#pragma unroll 1
                for (int c = part * 8; c < kt; c += epi_w * 8) {
                    unsigned v1[16], v2[16], w[4];             // HH | X1, X2 | LL
                    tmem_ld16(d1 + 2 * c, v1);
                    tmem_ld16(d2 + 2 * c, v2);
                    const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(bias + c);
                    const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(bias + c + 4);
                    unsigned long long y[4] = {b0.x, b0.y, b1.x, b1.y};
                    if (has_res) {
                        uint2 rh = make_uint2(0, 0), rl = rh;
                        if (live) {
                            const uint2* v = reinterpret_cast<const uint2*>(rsd + (c >> 4) * res_grp) + (c >> 3 & 1);
                            rh = v[0];
                            rl = v[2 * res_plane];
                        }
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const unsigned vh = i ? rh.y : rh.x, vl = i ? rl.y : rl.x;
                            const unsigned a = __byte_perm(vl, vh, 0x5140), b = __byte_perm(vl, vh, 0x7362);
                            y[2 * i] = fma2(pack2((float)(short)(a & 0xffffu), (float)((int)a >> 16)), r, y[2 * i]);
                            y[2 * i + 1] = fma2(pack2((float)(short)(b & 0xffffu), (float)((int)b >> 16)), r, y[2 * i + 1]);
                        }
                    }
                    tmem_ld_wait();
                    if (c + epi_w * 8 >= kt) {                 // the set may be filled again
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) count_up(&drained[set], nsets);
                    }
                    const float fixf = 128.0f * (float)(int)(s_hi * 256u + s_lo);
                    const unsigned long long fix = pack2(fixf, fixf);
                    if (short_sum) finish8<true>(v1, v2, fix, f, y, w);
                    else finish8<false>(v1, v2, fix, f, y, w);
#pragma unroll
                    for (int j = 0; j < 4; ++j) w[j] = __vmaxs2(w[j], floor2);
                    if (live) {
                        smx = __vmaxs2(__vmaxs2(smx, w[0]), __vmaxs2(__vmaxs2(w[1], w[2]), w[3]));
                        smn = __vmins2(__vmins2(smn, w[0]), __vmins2(__vmins2(w[1], w[2]), w[3]));
                    }
                    if (has_out && live) {
                        uint2* v = reinterpret_cast<uint2*>(dst + (c >> 4) * out_grp) + (c >> 3 & 1);
                        v[0] = make_uint2(__byte_perm(w[0], w[1], 0x7531), __byte_perm(w[2], w[3], 0x7531));
                        v[2 * out_plane] = make_uint2(__byte_perm(w[0], w[1], 0x6420), __byte_perm(w[2], w[3], 0x6420));
                    }
                    if (store && live && ok)
                        store8(store + ((long long)c * P * Q + h * Q + q) * p.N + n0 + img, (long long)P * Q * p.N, w[0], w[1], w[2], w[3]);
                }
                fence_async();
                __syncwarp();
                ++stored_tiles;
                if (lane == 0) publish(&done[slot * 4 + quarter], stored_tiles);
                for (tc += nsets; tc >= tcols; ++tr) tc -= tcols;
            }
            // the sets of other warps: their phases of this layer
            for (int s = 0; s < nsets; ++s)
                if (s != set && (((tiles - s + nsets - 1) / nsets) & 1) && s < tiles) full_bits ^= 1u << s;
            const int most = max((int)(short)smx, (int)smx >> 16), least = min((int)(short)smn, (int)smn >> 16);
            const int stat = __reduce_max_sync(0xffffffffu, max(most, -least));
            if (lane == 0 && stat) atomicMax(p.stats + L.slot_out, stat);
        }
        if (p.pooled) {
            // averages of the last layer's images, from what it has left in shared memory: a thread has an
            // image, a group of four channels and every 16th pixel (sums of up to 512 mantissas: exact)
            epilogue_barrier();
            const Layer& L = p.layer[p.n - 1];
            const int jobs = L.K / 4 << glog, pixels = L.P * L.Q;
            for (int i = threadIdx.x >> 4; i < jobs; i += kEpiWarps * 2) {
                const int g = i & (G - 1), c4 = i >> glog;
                int sum[4] = {0, 0, 0, 0};
                for (int px = threadIdx.x & 15; px < pixels; px += 16) {
                    const int h = px / L.Q, w = px - h * L.Q;
                    const unsigned* v = reinterpret_cast<const unsigned*>(smem) +
                                        (pixel_at(L.out, glog, h, g, w) + (c4 >> 2) * L.out.grp) * 4 + (c4 & 3);
                    const unsigned hi = v[0], lo = v[L.out.plane * 4];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        sum[k] += ((int)(hi << (24 - 8 * k)) >> 24) * 256 + (int)(lo >> 8 * k & 255u);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    for (int o = 8; o > 0; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
                if ((threadIdx.x & 15) == 0 && g < n_img && ok)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        p.pooled[(long long)(c4 * 4 + k) * p.N + n0 + g] = (short)__float2int_rn((float)sum[k] / (float)pixels);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kEpiWarps + 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
    if (threadIdx.x == 0 && *fail_flag && p.status) atomicExch(p.status, 1);
}

// ---- filters ---------------------------------------------------------------------------------------
// Filters C,R,S,K -> per layer [chunk][row of 16 bytes]: for every eight output channels eight rows with the
// high bytes of a chunk's 16 input channels and eight with their low bytes minus 128 (so that the epilogue
// finds what it adds up side by side: a load of tensor memory costs about as much for eight columns as for
// sixteen), row 2K ones (the sum of the activations).  Channels beyond C, the chunk that pads an odd number and the rows up to n2 are zero.
struct FilterJob {
    const short* F;
    long long at;
    int C, RS, K, n2, chunks;
    unsigned short chunk[2 * kStepsMost];    // tap * 256 + channel group; 0xffff: none
};
constexpr int kFilterJobs = 16;
struct FilterJobList { int n; FilterJob job[kFilterJobs]; };

__global__ void __launch_bounds__(256)
chain_filters_kernel(const __grid_constant__ FilterJobList list, unsigned char* __restrict__ planes) {
    after_earlier_kernels();
    const FilterJob& f = list.job[blockIdx.y];
    unsigned char* d = planes + f.at;
    const int total = f.chunks * f.n2 * 16;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int b = i & 15, row = (i >> 4) % f.n2, ch = (i >> 4) / f.n2;
        const unsigned id = f.chunk[ch];
        const int c = (int)(id & 255u) * 16 + b;
        unsigned char v = 0;
        if (id != 0xffffu && c < f.C && row <= 2 * f.K) {
            if (row == 2 * f.K) {
                v = 1;
            } else {
                const int k = (row >> 4) * 8 + (row & 7);
                const int m = (int)f.F[((long long)c * f.RS + (int)(id >> 8)) * f.K + k];
                v = (unsigned char)(row & 8 ? (m & 255) - 128 : m >> 8);
            }
        }
        d[i] = v;
    }
}

// ---- plan ------------------------------------------------------------------------------------------
inline int floor_half(int a) { return a >= 0 ? a / 2 : -((-a + 1) / 2); }

struct Tensor {
    int C, H, W;
    int top = 0, left = 0, maxh, maxw, parity = -1;      // what its readers reach; parity -1: none reads it
    int first, last = -2;                                // layers that write and last read it
    bool wanted = false;
    int at = -1, units = 0;
    Place place;                                         // relative to `at` until that is known
};

struct Region { int at, units, first, last; const Tensor* t; };

// One or two images to a CTA; false where the layers do not fit.
bool plan_for(const b2_conv_chain_layer* in, int n, int glog, unsigned high, Chain* out, std::vector<FilterJob>* jobs,
              size_t* filter_bytes, int* shapes, long long* ahead) {
    const int G = 1 << glog;
    std::vector<Tensor> ts(n + 1);                       // [0] the input, [l + 1] the result of layer l
    for (int l = 0; l < n; ++l) {
        const b2_conv_dims& d = in[l].dims;
        if (d.D != 1 || d.T != 1 || d.M != 1 || d.pad_d != 0 || d.dil_h != 1 || d.dil_w != 1) return false;
        if (d.str_h != d.str_w || d.str_h < 1 || d.str_h > 2 || d.R > 7 || d.S > 7 || d.R < 1 || d.S < 1) return false;
        if (d.pad_h < 0 || d.pad_w < 0 || d.pad_h > 3 || d.pad_w > 3) return false;
        if (d.K % 16 != 0 || d.K > kChannelsMost || d.K < 16 || d.C < 1 || d.C > 128) return false;
        if (d.H < 1 || d.W < 1 || d.P < 1 || d.Q < 1 || d.H > 128 || d.W > 128 || d.P > 128 || d.Q > 128) return false;
        if (d.N != in[0].dims.N || d.N < 1) return false;
        if (in[l].input < -1 || in[l].input >= l || in[l].residual < B2_CONV_CHAIN_NONE || in[l].residual >= l) return false;
        Tensor& x = ts[in[l].input + 1];
        if (l == 0 && in[l].input != -1) return false;
        if (l == 0) { x.C = d.C; x.H = d.H; x.W = d.W; x.first = -1; x.maxh = d.H - 1; x.maxw = d.W - 1; x.wanted = true; }
        if (x.C != d.C || x.H != d.H || x.W != d.W) return false;
        const int par = d.str_h == 2 ? 1 : 0;
        if (x.parity >= 0 && x.parity != par) return false;          // read at both strides
        x.parity = par;
        x.top = std::max(x.top, d.pad_h); x.left = std::max(x.left, d.pad_w);
        x.maxh = std::max(x.maxh, (d.P - 1) * d.str_h - d.pad_h + d.R - 1);
        x.maxw = std::max(x.maxw, (d.Q - 1) * d.str_w - d.pad_w + d.S - 1);
        x.last = l; x.wanted = true;
        if (in[l].residual >= -1) {
            Tensor& r = ts[in[l].residual + 1];
            if (r.C != d.K || r.H != d.P || r.W != d.Q) return false;
            r.last = std::max(r.last, l); r.wanted = true;
        }
        Tensor& y = ts[l + 1];
        y.C = d.K; y.H = d.P; y.W = d.Q; y.first = l; y.maxh = d.P - 1; y.maxw = d.Q - 1;
    }
    ts[n].wanted = true; ts[n].last = n;                 // (its averages are taken from there)
    // tensors of one shape have one layout, whatever their readers reach: they take over each other's
    // memory without new rings of zeros, and a layer may follow the one before tile by tile
    for (Tensor& t : ts) t.parity = std::max(t.parity, 0);
    for (Tensor& t : ts)
        for (const Tensor& o : ts) {
            if (!o.wanted || o.parity != t.parity || o.H != t.H || o.W != t.W || (o.C + 15) / 16 != (t.C + 15) / 16) continue;
            t.top = std::max(t.top, o.top); t.left = std::max(t.left, o.left);
            t.maxh = std::max(t.maxh, o.maxh); t.maxw = std::max(t.maxw, o.maxw);
        }
    for (Tensor& t : ts) {
        Place& p = t.place;
        p.parity = t.parity;
        const int groups = (t.C + 15) / 16;
        if (!t.parity) {
            p.pitch = t.W + std::max(t.left, t.maxw - (t.W - 1));
            p.off[0] = p.off[1] = p.off[2] = p.off[3] = t.top * G * p.pitch + t.left;
            p.grp = (t.top + t.maxh + 1) * G * p.pitch + t.left - (p.pitch - t.maxw - 1);
        } else {
            p.pitch = 1;
            for (int b = 0; b < 2; ++b) {
                const int data = floor_half(t.W - 1 - b) + 1, lo = floor_half(t.left + b), hi = floor_half(t.maxw - b) + 1;
                p.pitch = std::max(p.pitch, data + std::max(lo, hi - data));
            }
            int at = 0;
            for (int a = 0; a < 2; ++a)
                for (int b = 0; b < 2; ++b) {
                    const int lo_h = floor_half(t.top + a), lo_w = floor_half(t.left + b);
                    const int cols = std::max(floor_half(t.W - 1 - b), floor_half(t.maxw - b)) + 1;
                    p.off[2 * a + b] = at + lo_h * G * p.pitch + lo_w;
                    at += (lo_h + floor_half(t.maxh - a) + 1) * G * p.pitch + lo_w - (p.pitch - cols);
                }
            p.grp = at;
        }
        p.plane = groups * p.grp;
        t.units = 2 * p.plane;
    }
    const int room = kSmemMost / 16 - kFixedUnits;
    std::vector<Region> used;
    // the lowest place, or the highest
    auto fits = [&](int units, int first, int last, bool top) -> int {
        std::vector<std::pair<int, int>> busy;
        for (const Region& r : used)
            if (r.first <= last && first <= r.last) busy.push_back({r.at, r.at + r.units});
        std::sort(busy.begin(), busy.end());
        int at = 0, found = -1;
        for (const auto& b : busy) {
            if (b.first - at >= units) { found = top ? b.first - units : at; if (!top) return found; }
            at = std::max(at, b.second);
        }
        if (room - at >= units) found = top ? room - units : at;
        return found;
    };
    auto same_layout = [](const Tensor& a, const Tensor& b) {
        return a.parity == b.parity && a.units == b.units && a.H == b.H && a.W == b.W && a.place.pitch == b.place.pitch &&
               a.place.grp == b.place.grp && a.place.off[0] == b.place.off[0] && a.place.off[3] == b.place.off[3] &&
               a.top == b.top && a.left == b.left && a.maxh == b.maxh && a.maxw == b.maxw;
    };
    // activations first, those of the i-th shape as high as they fit where bit i of `high` is set; a result takes the place of the residual that it adds where that is its last reader
    std::vector<const Tensor*> kinds;
    for (int i = 0; i <= n; ++i) {
        Tensor& t = ts[i];
        if (!t.wanted) continue;
        int kind = 0;
        while (kind < (int)kinds.size() && !same_layout(*kinds[kind], t)) ++kind;
        if (kind == (int)kinds.size()) kinds.push_back(&t);
        const int l = i - 1, r = l >= 0 ? in[l].residual : B2_CONV_CHAIN_NONE;
        if (r >= -1 && ts[r + 1].last == l && same_layout(t, ts[r + 1]) && in[l].input != r) {
            t.at = ts[r + 1].at;
        } else {
            t.at = fits(t.units, t.first, t.last, high >> kind & 1u);
            if (t.at < 0) return false;
        }
        used.push_back({t.at, t.units, t.first, t.last, &t});
    }
    Chain& c = *out;
    c.n = n; c.glog = glog; c.N = in[0].dims.N; c.inC = ts[0].C; c.inH = ts[0].H; c.inW = ts[0].W;
    auto placed = [](const Tensor& t) {
        Place p = t.place;
        for (int i = 0; i < 4; ++i) p.off[i] += t.at;
        return p;
    };
    c.in = placed(ts[0]);
    size_t bytes = 0;
    int top_unit = 0;
    for (int l = 0; l < n; ++l) {
        const b2_conv_dims& d = in[l].dims;
        Layer& L = c.layer[l];
        const Tensor &x = ts[in[l].input + 1], &y = ts[l + 1];
        // chunks of 16 input channels under a tap, by address; two of them make a k-step
        struct Chunk { int at, tap, group; };
        std::vector<Chunk> ch;
        const int groups = (d.C + 15) / 16;
        for (int g = 0; g < groups; ++g)
            for (int r = 0; r < d.R; ++r)
                for (int s = 0; s < d.S; ++s) {
                    const int h = r - d.pad_h, w = s - d.pad_w;
                    const int a = x.parity ? x.place.off[(h & 1) * 2 + (w & 1)] + floor_half(h) * G * x.place.pitch + floor_half(w)
                                           : x.place.off[0] + h * G * x.place.pitch + w;
                    if (a < 0) return false;
                    ch.push_back({a + g * x.place.grp, r * d.S + s, g});
                }
        std::sort(ch.begin(), ch.end(), [](const Chunk& a, const Chunk& b) { return a.at < b.at; });
        L.nk = ((int)ch.size() + 1) / 2;
        if (L.nk > kStepsMost) return false;
        FilterJob job;
        job.F = in[l].filters; job.C = d.C; job.RS = d.R * d.S; job.K = d.K; job.chunks = 2 * L.nk;
        L.K = d.K; L.P = d.P; L.Q = d.Q;
        L.n2 = (2 * d.K + 1 + 15) / 16 * 16;
        L.nsets = 8 * L.n2 <= 512 ? 4 : 4 * L.n2 <= 512 ? 2 : 1;
        job.n2 = L.n2; job.at = (long long)bytes;
        int reach = 0;
        for (int k = 0; k < L.nk; ++k) {
            const Chunk& a = ch[2 * k];
            const bool pair = 2 * k + 1 < (int)ch.size();
            const int dist = pair ? ch[2 * k + 1].at - a.at : 1;
            if (dist < 1) return false;
            L.step[k] = (unsigned)a.at | (unsigned)dist << 16;
            job.chunk[2 * k] = (unsigned short)(a.tap << 8 | a.group);
            job.chunk[2 * k + 1] = pair ? (unsigned short)(ch[2 * k + 1].tap << 8 | ch[2 * k + 1].group) : 0xffff;
            reach = std::max(reach, a.at + dist);
        }
        jobs->push_back(job);
        L.filt_src = (long long)bytes;
        L.filt_units = L.nk * 2 * L.n2;
        bytes += (size_t)L.filt_units * 16;
        L.a_base = x.at; L.sbo = x.place.pitch; L.a_row = 16 * x.place.pitch; L.plane = x.place.plane;
        L.tcols = (d.Q + 7) / 8; L.trows = (d.P * G + 15) / 16; L.tiles = L.tcols * L.trows;
        if (L.tiles > kTilesMost) return false;
        // how far the last tile's instructions read (rows and columns that do not exist included)
        top_unit = std::max(top_unit, x.at + x.place.plane + reach + (L.trows - 1) * L.a_row + (L.tcols - 1) * 8 +
                                          15 * x.place.pitch + 8);
        L.has_out = y.wanted ? 1 : 0;
        L.has_res = in[l].residual >= -1 ? 1 : 0;
        L.out = y.wanted ? placed(y) : c.in;
        L.res = L.has_res ? placed(ts[in[l].residual + 1]) : c.in;
        L.slot_in = in[l].slot_in; L.slot_f = in[l].slot_filters; L.slot_out = in[l].slot_out;
        L.slot_bias = in[l].slot_bias; L.slot_res = in[l].slot_residual;
        L.relu = in[l].relu ? 1 : 0;
        // 256*HH + X fits 32 bits, and the tile kernel's variant for whole blocks of images takes it as one
        // number (the last bit of the fp32 sum depends on it)
        L.short_sum = (long long)d.C * d.R * d.S * ((1 << 22) + (1 << 16)) < (1LL << 31) && d.N % 128 == 0 &&
                      (long long)d.K * d.P * d.Q * d.N < (1LL << 32);
        L.bias = in[l].bias; L.dst = in[l].out;
    }
    // filters: ahead of their layer where there is room for them beside what is live then
    for (int l = 0; l < n; ++l) {
        Layer& L = c.layer[l];
        L.prefetch = 1;
        L.filt = fits(L.filt_units, l - 1, l, false);
        if (L.filt < 0) { L.prefetch = 0; L.filt = fits(L.filt_units, l, l, false); }
        if (L.filt < 0) return false;
        *ahead += L.prefetch ? L.filt_units : 0;
        used.push_back({L.filt, L.filt_units, l - L.prefetch, l, nullptr});
    }
    int end = top_unit;
    for (const Region& r : used) end = std::max(end, r.at + r.units);
    if (end > room) return false;
    c.smem_units = end;
    *filter_bytes = bytes;
    // Which layers may follow the one before tile by tile, and which results need their zero ring made.
    // Tile by tile: the layer reads the result of the one before at the same geometry, and stores into
    // memory that the layer before may still use only in ways that concern the same pixels -- as the
    // operand, whose readers are the tiles that this one has waited for, or as the residual.
    for (int l = 0; l < n; ++l) {
        Layer& L = c.layer[l];
        const b2_conv_dims& d = in[l].dims;
        const Tensor& y = ts[l + 1];
        L.zero = 0; L.zero_at = 0; L.zero_units = 0;
        if (y.wanted) {
            // the last tensor of this layout that lay here left its ring of zeros; what came after it,
            // or what has been here at all, did not
            const bool in_place = in[l].residual >= -1 && ts[in[l].residual + 1].at == y.at && ts[in[l].residual + 1].last == l;
            int since = -2;
            for (const Region& r : used)
                if (r.t && r.t != &y && r.first < l && r.at == y.at && same_layout(*r.t, y)) since = std::max(since, r.first);
            for (const Region& r : used) {
                if (r.t == &y || r.first >= l || r.first <= since || r.at >= y.at + y.units || y.at >= r.at + r.units) continue;
                if (!in_place) L.zero = 1;
            }
        }
        if (L.zero) { L.zero_at = y.at; L.zero_units = y.units; }
        bool fine = l > 0 && in[l].input == l - 1 && d.str_h == 1 && !L.zero && !c.layer[l - 1].zero &&
                    d.P == in[l - 1].dims.P && d.Q == in[l - 1].dims.Q && L.n2 == c.layer[l - 1].n2 &&
                    d.R - 1 <= 7 && d.pad_w <= 7 && d.pad_h * G <= 15 && (d.R - 1 - d.pad_h) * G <= 15 && L.tcols >= 1;
        if (fine && y.wanted)
            for (const Region& r : used) {
                if (r.t == &y || r.last < l - 2 || r.last >= l || r.at >= y.at + y.units || y.at >= r.at + r.units) continue;
                if (!(r.t && r.at == y.at && same_layout(*r.t, y))) fine = false;
            }
        L.coarse = fine ? 0 : 1;
        *ahead += fine ? 256 : 0;
    }
    *shapes = (int)kinds.size();
    return true;
}

// The plan of a chain: two images to a CTA where one would make more CTAs than there are SMs (a layer of two
// images takes 1.4 times one of one: filters are read once for both, and 64 pixels of each fill an
// instruction's rows), one elsewhere, or where two do not fit.
bool plan(const b2_conv_chain_layer* in, int n, Chain* out, std::vector<FilterJob>* jobs, size_t* filter_bytes) {
    if (n < 1 || n > kLayersMost) return false;
    for (int glog = in[0].dims.N > 148 ? 1 : 0; glog >= 0; --glog) {
        // Which shapes lie high decides what is left in one piece for the filters: the arrangement that
        // takes most of them in ahead of time (a 64-channel layer's are 83 KB: 2 us when waited for).
        long long best = -1;
        unsigned which = 0;
        int shapes = 1;
        for (unsigned high = 0; high < 1u << std::min(shapes, 6); ++high) {
            long long ahead = 0;
            jobs->clear();
            if (plan_for(in, n, glog, high, out, jobs, filter_bytes, &shapes, &ahead) && ahead > best) { best = ahead; which = high; }
        }
        if (best < 0) continue;
        long long ahead = 0;
        jobs->clear();
        return plan_for(in, n, glog, which, out, jobs, filter_bytes, &shapes, &ahead);
    }
    return false;
}

// Whether the chain is the faster way (microseconds, both sides as measured on ResNets of 10 to 22 layers, 8x8
// to 32x32 pixels, 1 to 2048 images).  The chain: a start of 8, then per layer the hand-overs between its
// roles and 0.25 a tile -- once per wave of 148 blocks --, and its stores of results that somebody outside
// reads go to a line each.  One by one: 6 a launch and 1.46e-6 a result, in blocks of 128 images.  22 layers
// of ResNet-20: 1 image 83 against 175, 100 images 85 / 159 (n = 64), 256 images 120 / 204, 300 images (two
// waves) 234 / 429, 512 images 237 / 310, 2048 images 828 / 970; ten layers on 16x16 pixels, 1024 images
// (four waves): 130 / 89, and two layers on 32x32 pixels, 256 images, the second stored: 38 / 21.
bool faster(const b2_conv_chain_layer* in, const Chain& c) {
    double chain = 8.0, stores = 0.0, apart = 0.0;
    for (int l = 0; l < c.n; ++l) {
        const b2_conv_dims& d = in[l].dims;
        const double results = (double)d.K * d.P * d.Q;
        chain += 3.2 + 0.25 * c.layer[l].tiles;
        if (in[l].out) stores += 0.0006 * results * (1 << c.glog);
        apart += 6.0 + 1.46e-6 * results * ((d.N + 127) / 128 * 128);
    }
    const int blocks = (c.N + (1 << c.glog) - 1) >> c.glog;
    return (double)((blocks + 147) / 148) * (chain + stores) < apart;
}

}  // namespace

extern "C" int b2_conv_chain_info(const b2_conv_chain_layer* layers, int32_t n, int32_t* supported,
                                  size_t* filter_bytes) {
    B2_REQUIRE(layers && n >= 1 && supported && filter_bytes, "null argument");
    std::vector<Chain> c(1);
    std::vector<FilterJob> jobs;
    *filter_bytes = 0;
    *supported = plan(layers, n, &c[0], &jobs, filter_bytes) && faster(layers, c[0]) ? 1 : 0;
    return B2_OK;
}

extern "C" int b2_conv_chain_filters(const b2_conv_chain_layer* layers, int32_t n, void* filter_planes,
                                     int32_t* launches, void* stream) {
    B2_REQUIRE(layers && n >= 1 && filter_planes && launches, "null argument");
    B2_REQUIRE(((uintptr_t)filter_planes & 15) == 0, "filter planes must be 16-byte aligned");
    std::vector<Chain> c(1);
    std::vector<FilterJob> jobs;
    size_t bytes;
    B2_REQUIRE(plan(layers, n, &c[0], &jobs, &bytes), "these layers do not make a chain");
    *launches = 0;
    for (size_t i = 0; i < jobs.size(); i += kFilterJobs) {
        FilterJobList list;
        list.n = (int)std::min<size_t>(kFilterJobs, jobs.size() - i);
        for (int j = 0; j < list.n; ++j) {
            B2_REQUIRE(jobs[i + j].F, "null filters");
            list.job[j] = jobs[i + j];
        }
        B2_CUDA(b2::launch_after(chain_filters_kernel, dim3(32, (unsigned)list.n), 256, 0, (cudaStream_t)stream, list,
                                 (unsigned char*)filter_planes));
        ++*launches;
    }
    return B2_OK;
}

extern "C" int b2_conv_chain_flex16(const b2_conv_chain_layer* layers, int32_t n, const int16_t* x,
                                    const void* x_planes, size_t plane_bytes, const void* filter_planes,
                                    const b2_flex_scale* table, int32_t* stats, int16_t* pooled, int32_t* status,
                                    void* stream) {
    B2_REQUIRE(layers && n >= 1 && (x || x_planes) && filter_planes && table && stats, "null argument");
    B2_REQUIRE(((uintptr_t)filter_planes & 15) == 0, "filter planes must be 16-byte aligned");
    std::vector<Chain> keep(1);
    Chain& c = keep[0];
    std::vector<FilterJob> jobs;
    size_t bytes;
    B2_REQUIRE(plan(layers, n, &c, &jobs, &bytes), "these layers do not make a chain");
    for (int l = 0; l < n; ++l)
        B2_REQUIRE(layers[l].slot_in >= 0 && layers[l].slot_filters >= 0 && layers[l].slot_out >= 0 &&
                   (!layers[l].bias || layers[l].slot_bias >= 0) && (layers[l].residual < -1 || layers[l].slot_residual >= 0),
                   "a layer's scale slots are missing");
    if (x) {
        c.src_lo = (const unsigned char*)x; c.src_hi = c.src_lo + 1;
        c.src_pitch = 2LL * c.N; c.src_estep = 2;
    } else {
        c.src_hi = (const unsigned char*)x_planes; c.src_lo = c.src_hi + plane_bytes;
        c.src_pitch = (c.N + 15) / 16 * 16; c.src_estep = 1;
    }
    c.filters = (const unsigned char*)filter_planes; c.table = table; c.stats = stats; c.status = status;
    c.pooled = pooled;
    B2_REQUIRE(!pooled || layers[n - 1].dims.P * layers[n - 1].dims.Q <= 512, "too many pixels to average");
    static bool attr_set = false;
    if (!attr_set) {
        B2_CUDA(cudaFuncSetAttribute(conv_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMost));
        attr_set = true;
    }
    const size_t smem = ((size_t)c.smem_units + kFixedUnits) * 16;
    B2_CUDA(b2::launch_after(conv_chain_kernel, dim3((unsigned)((c.N + (1 << c.glog) - 1) >> c.glog)), kCtaThreads, smem,
                             (cudaStream_t)stream, c));
    return B2_OK;
}
