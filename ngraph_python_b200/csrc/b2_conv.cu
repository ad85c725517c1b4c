// Convolution forward (and average pooling) for tensors in the reference's C,D,H,W,N layout.
//
// Takes the place of ConvFpropKernel / FlexConvFpropKernel and the direct-convolution SASS they
// select (ngraph/transformers/gpu/conv.py:24-100, gpu/flex_conv.py:49-200,
// gpu/kernels/sass/?conv_xprop_*.sass), and of the avg-pooling forward kernel
// (gpu/pool.py:27-220, gpu/kernels/cuda/pooling.py:291-438).
//
// fprop:  O[K,M,P,Q,N] = sum_{c,t,r,s} F[C,T,R,S,K] * I[C,D,H,W,N]
// is run as one GEMM on the tensor cores, O^T[(p,q,n), k] = Icol[(p,q,n),(c,r,s)] * F[(c,r,s), k].  flex16
// takes the tile kernel below (byte planes, windows fetched by TMA), fp32 and dilated filters the product
// that gathers its operands on the way in (b2_direct.cuh); what neither takes (depth, large windows)
// goes through memory:
//   * a gather pre-pass writes the rows of Icol (one row per output pixel and image, the filter
//     window unrolled along K, zero where the window hangs over the border) directly as the two
//     operand planes the GEMM kernel streams with TMA (int8 hi/lo for flex16, tf32 hi/lo for
//     fp32), so the input is read once and no separate split pass is needed;
//   * the filter planes come from the same split kernel the GEMM uses (F is already [(c,r,s)][k]);
//   * the tile kernel's epilogue stores column-major, which is exactly the K,P,Q,N layout: for a
//     fixed output channel the 32 lanes of a warp hold 32 consecutive images -> coalesced stores.
// N (batch) is the GEMM-M direction (128 rows per tile), the output channels are the GEMM-N
// direction with a 16/32/64/128-wide tile, so the small channel counts of ResNet-20 do not pad
// the tensor-core tile to 128.
//
// The two training contractions (ConvBpropKernel / ConvUpdateKernel, gpu/conv.py:121-312,
// FlexConvBpropKernel / FlexConvUpdateKernel, gpu/flex_conv.py:203-621; readable specification
// ngraph/transformers/cpu/cpuengine.py:256-271 and :395-418) have the same three ways; through
// memory:
//   bprop:  gI^T[(h,w,n), c] = Ecol[(h,w,n),(k,r,s)] * F[(c,r,s),k] read as [(k,r,s)][c], where the
//           gather takes E[k,p,q,n] with p = (h + pad - r*dil) / str when that division is exact
//           and p lies inside the output, zero otherwise (the transposed, flipped convolution);
//   update: U[(c,r,s), k] = Icol^T[(c,r,s),(p,q,n)] * E[k,(p,q,n)]: the contraction runs over all
//           output positions and images (262144 for a 32x32 layer at batch 256), so it is cut
//           into K slices spread over the SMs; the slices are added in a fixed order by a second
//           kernel (deterministic, and exact for flex16: every slice is an exact integer).
#include <cstdlib>

#include "b2_direct.h"
#include "b2_gemm_impl.cuh"

namespace {

struct ConvGeom {
    int C, H, W, N, K, R, S, P, Q, pad_h, pad_w, str_h, str_w, dil_h, dil_w;
    // depth (the reference's D / T / M axes): handled by the gather + GEMM path only; the tile
    // kernels take convolutions with D = T = M = 1
    int D, T, M, pad_d, str_d, dil_d;
    // the tile kernel's view of an input gradient: C, H, W are the error tensor's, K, P, Q the input's,
    // the rest the forward convolution's
    int bprop;
};

// Byte planes have their rows of N images padded to a multiple of 16 bytes (what TMA strides need).
inline int plane_pitch(int n) { return (n + 15) / 16 * 16; }
inline size_t plane_size(int c, int h, int w, int n) {
    return ((size_t)c * h * w * plane_pitch(n) + 1023) / 1024 * 1024;
}
inline int image_blocks(int n) { return (n + 127) / 128; }

int geom_from(const b2_conv_dims* d, ConvGeom* g) {
    B2_REQUIRE(d, "null dims");
    B2_REQUIRE(d->C > 0 && d->H > 0 && d->W > 0 && d->N > 0 && d->K > 0 && d->R > 0 && d->S > 0 &&
               d->P > 0 && d->Q > 0 && d->str_h > 0 && d->str_w > 0 && d->dil_h > 0 && d->dil_w > 0 &&
               d->D > 0 && d->T > 0 && d->M > 0 && d->str_d > 0 && d->dil_d > 0 && d->pad_d >= 0 &&
               d->pad_h >= 0 && d->pad_w >= 0,
               "bad convolution dimensions");
    B2_REQUIRE((long long)d->D * d->H * d->W < (1 << 24) && (long long)d->M * d->P * d->Q < (1 << 24),
               "convolution extents too large");
    g->C = d->C; g->H = d->H; g->W = d->W; g->N = d->N; g->K = d->K; g->R = d->R; g->S = d->S;
    g->P = d->P; g->Q = d->Q; g->pad_h = d->pad_h; g->pad_w = d->pad_w; g->str_h = d->str_h;
    g->str_w = d->str_w; g->dil_h = d->dil_h; g->dil_w = d->dil_w;
    g->bprop = 0;
    g->D = d->D; g->T = d->T; g->M = d->M; g->pad_d = d->pad_d; g->str_d = d->str_d;
    g->dil_d = d->dil_d;
    return B2_OK;
}

inline bool flat_depth(const ConvGeom& g) {
    return g.D == 1 && g.T == 1 && g.M == 1 && g.pad_d == 0;
}

inline int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

// One direction of a tile's window: output positions tile*g .. tile*g + g-1, filter extent r.
//   forward:        input = out * str - pad + tap
//   input gradient: error = (out + pad - tap) / str where that divides; g is a multiple of str, so every
//                   tile has the same residues and steps g / str errors further
inline void window(int bprop, int g, int r, int pad, int str, int* extent, int* off, int* step) {
    if (!bprop) {
        *extent = (g - 1) * str + r; *off = -pad; *step = g * str;
    } else {
        const int lo = -floor_div(-(pad - r + 1), str), hi = floor_div(g - 1 + pad, str);
        *extent = hi - lo + 1 > 1 ? hi - lo + 1 : 1; *off = lo; *step = g / str;
    }
}

// The arguments without the tensors of a pass (0 forward, 1 input gradient) for the kernel that gathers
// and converts its operands on the way in (b2_direct.cuh), with gh x gw pixels to a row of the product;
// false where a tile does not fit the convolution.  One pixel: every value of a window is gathered and
// converted once per tap.  Several: the window they share is gathered once (2x2 pixels under 3x3
// filters: 4 values a pixel and channel instead of 9) against filters padded with zeros, and as many
// times fewer rows of the product fill the machine in one wave (16 channels, 32x32, batch 100: 800
// tiles of 128 rows before).  The input gradient of a strided convolution needs tiles that are multiples
// of the stride, in which every pixel finds its own residue class of taps.
inline bool direct_args(int mode, const ConvGeom& g, int pass, int gh, int gw, b2_direct_args* out) {
    const bool tiled = gh * gw > 1, strided = g.str_h > 1 || g.str_w > 1;
    const int result = pass ? g.C : g.K, read = pass ? g.K : g.C;         // channels
    const int rp = pass ? g.H : g.P, rq = pass ? g.W : g.Q;               // extents of the result
    if (tiled && (g.dil_h != 1 || g.dil_w != 1 || result % 8 != 0)) return false;
    if (pass && strided && (gh % g.str_h != 0 || gw % g.str_w != 0)) return false;
    b2_direct_args d = {};
    d.flex = mode == MODE_FLEX16;
    d.a_kind = B2_OPERAND_GATHER;
    b2_gather& t = d.g;
    t.channels = read; t.H = pass ? g.P : g.H; t.W = pass ? g.Q : g.W; t.N = g.N;
    t.P = (rp + gh - 1) / gh; t.Q = (rq + gw - 1) / gw;
    t.channel_last = pass;
    if (tiled) {
        window(pass, gh, g.R, g.pad_h, g.str_h, &t.R, &t.off_h, &t.step_h);
        window(pass, gw, g.S, g.pad_w, g.str_w, &t.S, &t.off_w, &t.step_w);
        t.tap_h = t.tap_w = 1;
        t.gh = gh; t.gw = gw; t.kt = result; t.out_p = rp; t.out_q = rq; t.fr = g.R; t.fs = g.S;
        t.f0_h = pass ? g.pad_h - g.str_h * t.off_h : 0; t.f0_w = pass ? g.pad_w - g.str_w * t.off_w : 0;
        t.f1_h = pass ? -g.str_h : 1; t.f1_w = pass ? -g.str_w : 1;
        t.f2_h = pass ? 1 : -g.str_h; t.f2_w = pass ? 1 : -g.str_w;
        d.b_kind = B2_OPERAND_FILTER;
        d.b_rs = pass ? (long long)g.R * g.S * g.K : 1;
        d.b_ks = pass ? 1 : (long long)g.R * g.S * g.K;
    } else {
        t.R = g.R; t.S = g.S; t.gh = t.gw = 1;
        t.off_h = pass ? g.pad_h : -g.pad_h; t.off_w = pass ? g.pad_w : -g.pad_w;
        t.step_h = g.str_h; t.step_w = g.str_w;
        t.tap_h = pass ? -g.dil_h : g.dil_h; t.tap_w = pass ? -g.dil_w : g.dil_w;
        d.b_kind = pass ? B2_OPERAND_K : B2_OPERAND_ROWS;
        d.b_rs = pass ? (long long)g.R * g.S * g.K : 1;
        d.b_ks = pass ? 1 : g.K;
    }
    const long long rows = (long long)t.P * t.Q * g.N, k = (long long)read * t.R * t.S;
    if (rows >= (1LL << 31) - 256 || k > 32768 || (long long)result * g.R * g.S * read >= (1LL << 31)) return false;
    d.M = (int)rows; d.N = gh * gw * result; d.K = (int)k;
    d.ldc = (long long)rp * rq * g.N; d.colmajor = 1;
    *out = d;
    return true;
}

// Cycles of the gather + GEMM path: the planes of the unrolled rows once out and once back (at 5 TB/s), then
// the tile kernel.
inline long long unrolled_cost(int mode, const ConvGeom& g, int pass) {
    const long long rows = pass ? (long long)g.H * g.W * g.N : (long long)g.P * g.Q * g.N;
    const long long k = (long long)(pass ? g.K : g.C) * g.R * g.S;
    if (rows >= (1LL << 31) - 256) return 1LL << 62;
    const Shapes s = shapes_for(mode, (int)rows, pass ? g.C : g.K, (int)k);
    const long long planes = rows * s.Kp * s.esize * 4 / 2600;
    const long long kb = (mode == MODE_FLEX16 ? 1430LL : 1100LL) * (128 + s.bn) / 256;
    const long long tiles = (long long)(s.Mp / kBlockM) * (s.Np / s.bn);
    return 13000 + planes + (tiles + 147) / 148 * (3500 + (long long)(s.Kp * s.esize / kKBytes) * kb);
}

// fp32: what a shape and tile of a pass may add up, whichever is taken: the k-blocks in one sum
// (b2_direct_args::longest), and where one block holds all of K no more than that one (further sums are added to
// nearest, which is nothing beside the blocks' loss but is something beside none: 16 -> 32 channels 1x1 at stride
// 2, batch 384, in three blocks of a 1x3 tile 1.09e-7 of the result's root mean square against 64 bits, 1.00e-7 in
// one).  An unrolled product adds chains of 16.
struct SumBound {
    int longest;
    bool one_block;
    bool allows(const b2_direct_args& d) const { return !one_block || d.K <= 32; }
};

inline SumBound sum_bound(int mode, const ConvGeom& g, int pass) {
    if (mode != MODE_F32X3) return {0, false};                    // (exact)
    long long best = -1;
    SumBound bound = {0, false};
    for (int a = 1; a <= 2; ++a)
        for (int b = 1; b <= 2; ++b) {
            b2_direct_args d;
            int n = 0;
            if (!direct_args(mode, g, pass, pass ? a * g.str_h : a, pass ? b * g.str_w : b, &d)) continue;
            const long long cost = b2_direct_longest(d, &n);
            if (cost < 0 || (best >= 0 && cost >= best)) continue;
            best = cost;
            bound = {n, d.K <= 32};
        }
    if (best >= 0 && best < unrolled_cost(mode, g, pass)) return bound;
    const int blocks = ((pass ? g.K : g.C) * g.R * g.S + 31) / 32;
    return {blocks < 16 ? blocks : 16, blocks == 1};
}

// Whether a pass goes that way, with the best tile.  It does what the gather + GEMM path does, with one
// launch and without writing the unrolled planes (8 bytes for each of the R*S copies of a value, and
// reading them again); the planes pay only where a long list of output channels would have the gather
// repeated for every 128 of them.
inline bool conv_goes_direct(int mode, const ConvGeom& g, int pass, b2_direct_args* out, SumBound* bound_out = nullptr) {
    if (!flat_depth(g) || getenv("B2_CONV_IM2COL")) return false;
    const SumBound bound = sum_bound(mode, g, pass);
    if (bound_out) *bound_out = bound;
    long long best = -1;
    for (int a = 1; a <= 2; ++a)
        for (int b = 1; b <= 2; ++b) {
            b2_direct_args d;
            if (!direct_args(mode, g, pass, pass ? a * g.str_h : a, pass ? b * g.str_w : b, &d) || !bound.allows(d)) continue;
            d.longest = bound.longest;
            const long long cost = b2_direct_cost(d);
            if (cost < 0 || (best >= 0 && cost >= best)) continue;
            best = cost;
            *out = d;
        }
    return best >= 0 && best < unrolled_cost(mode, g, pass);
}

// The same with the filters' rows made beforehand (b2_direct_stage_filters), for fp32 convolutions that go
// direct: false where a launch would take no less time (what the kernel's cost rule says for both; a row of
// filters costs its producers as much as a gathered one, or more).  With only the gathered rows to make, tiles
// of six pixels pay: 16 channels at 32x32, batch 100, 12.8 us against 16.7 for four, as they lie 20.2.
//
// Infinities and NaN: a row of the product holds the whole window of its tile, and a value outside a pixel's own
// taps meets zeros of that pixel's filters.  An infinity or NaN therefore makes every result of its image NaN that
// stands in a tile whose window covers it: up to 2x2 pixels with filters as they lie, 4x4 here (times the stride in
// an input gradient), beside those whose taps see it.  One-pixel tiles reach no further than the taps.
// `other`, unless NULL: what it would be without the kernel of b2_gather.cu.
inline bool conv_goes_staged(const ConvGeom& g, int pass, b2_direct_args* out, b2_direct_args* other = nullptr) {
    SumBound bound;
    if (!conv_goes_direct(MODE_F32X3, g, pass, out, &bound)) return false;
    long long best = b2_direct_cost(*out);
    b2_direct_args tile[16];
    int n = 0;
    bool found = false;
    for (int a = 1; a <= 4; ++a)
        for (int b = 1; b <= 4; ++b) {
            b2_direct_args& d = tile[n];
            if (!direct_args(MODE_F32X3, g, pass, pass ? a * g.str_h : a, pass ? b * g.str_w : b, &d) || !bound.allows(d)) continue;
            ++n;
            d.longest = bound.longest;
            d.staged = out;                       // (there will be such)
            d.staged_own = 1;
            const long long cost = b2_direct_cost(d);
            if (cost < 0 || cost >= best) continue;
            best = cost;
            found = true;
            *out = d;
        }
    if (other) *other = *out;
    if (g.N % 4 != 0) return found;
    // The kernel of b2_gather.cu, where it takes less.  It does not put more k-blocks into one sum of large terms (hi x
    // hi) than the one of b2_direct.cuh in the tile and shape that it would take, and its sums do not lose more: k-blocks
    // alone do not say it, those of 64 -> 64 channels at 8x8, batch 100, in tiles of one pixel are dense where a quarter
    // of 1x2 pixels' are zeros, in five slices of three and two (input gradient 2.04e-7 -> 2.18e-7 against 64 bits in two
    // slices of three and two; 32 -> 8 channels at 24x7, batch 220, 1.92e-7 -> 2.59e-7).  Shorter sums until that holds.
    // Sums of small terms have up to twice as many k-blocks as the large ones; they lose 2^-11 of what those do.
    const int longest = b2_direct_in_one_sum(*out);
    b2_gemm_plan_info plan;
    b2_direct_plan(*out, &plan);
    long long cost[16];
    double limit = -1;
    for (int i = 0; i < n; ++i) {
        tile[i].longest = longest;
        tile[i].staged_own = 0;
        cost[i] = b2_direct_cost(tile[i]);
    }
    for (;;) {
        int i = -1;
        for (int j = 0; j < n; ++j)
            if (cost[j] >= 0 && cost[j] < best && (i < 0 || cost[j] < cost[i])) i = j;
        if (i < 0) return found;
        // The same shape in more than one wave: two of the other kernel's CTAs share an SM and take less than its rule says
        // (3 <- 16 channels 3x3 at 32x32, batch 128, 28.9 us, 38.8 in this one; 32 <- 16 at stride 2, batch 200, 17.3 and 20.1).
        if (plan.waves > 1 && plan.tile_n < 128 && tile[i].g.gh == out->g.gh && tile[i].g.gw == out->g.gw && cost[i] > best - best / 5) {
            const b2_gather_info own = b2_gather_plan(tile[i]);
            if (own.bn == plan.tile_n && own.splits == plan.slices) return found;
        }
        if (limit < 0) limit = b2_direct_loss(*out) * (1 + 1e-9);
        if (b2_direct_loss(tile[i]) <= limit) {
            *out = tile[i];
            return true;
        }
        tile[i].longest = b2_direct_in_one_sum(tile[i]) - 1;
        cost[i] = tile[i].longest > 0 ? b2_direct_cost(tile[i]) : -1;
    }
}

inline int launch_direct(b2_direct_args& d, const void* A, const void* B, void* C,
                         const b2_flex_scale* table, int slotA, int slotB, int slotC, int* stats,
                         unsigned long long* probe_out, int* status, int probe, cudaStream_t st) {
    d.A = A; d.B = B; d.C = C; d.table = table; d.slotA = slotA; d.slotB = slotB; d.slotC = slotC;
    d.stats = stats; d.probe_out = probe_out; d.status = status; d.probe = probe;
    return b2_direct_launch(d, st);
}

// Gather + split.  Rows of the planes: r = ((m*P + p)*Q + q)*N + n ; columns:
// kidx = ((c*T + t)*R + r_)*S + s_.
// A block owns 32 consecutive rows (32 images of one output pixel when N is a multiple of 32) and
// walks the columns in chunks of 128 bytes of plane row.  Per chunk the tap decomposition of each
// column is computed once into shared memory; loads run along n (contiguous in the input), the
// write phase emits one 16-byte vector per thread and plane (contiguous along the plane row).
// BPROP = true gathers the rows of Ecol instead: row = (h*W + w)*N + n of the INPUT gradient,
// column = (k*R + r_)*S + s_, source E[k, p, q, n] (see the head of this file).
template <typename T, int MODE, bool BPROP>
__global__ void __launch_bounds__(256)
im2col_planes_kernel(const T* __restrict__ I, ConvGeom g, int rows, int kg, int rows_p, int kp,
                     void* __restrict__ plane0, void* __restrict__ plane1) {
    constexpr int CK = MODE == MODE_FLEX16 ? 128 : 32;
    __shared__ T tile[CK][33];
    __shared__ int tab_c[CK], tab_h[CK], tab_w[CK], tab_d[CK];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int r0 = blockIdx.x * 32;
    const int r = r0 + tx;
    const bool rvalid = r < rows;
    int n = 0, h0 = 0, w0 = 0, d0 = 0;
    if (rvalid) {
        n = r % g.N;
        const int pq = r / g.N;
        if (BPROP) {
            const int hw = pq % (g.H * g.W);
            d0 = pq / (g.H * g.W) + g.pad_d;
            h0 = hw / g.W + g.pad_h;
            w0 = hw % g.W + g.pad_w;
        } else {
            const int q = pq % g.Q, mp = pq / g.Q, pp = mp % g.P;
            d0 = (mp / g.P) * g.str_d - g.pad_d;
            h0 = pp * g.str_h - g.pad_h;
            w0 = q * g.str_w - g.pad_w;
        }
    }
    const int RS = g.R * g.S, TRS = g.T * RS;
    const int wr = threadIdx.x >> 3, vec = threadIdx.x & 7;
    const int orow = r0 + wr;
    for (int kc = 0; kc < kp; kc += CK) {
        __syncthreads();
        if (threadIdx.x < CK) {
            const int kidx = kc + threadIdx.x;
            if (kidx < kg) {
                const int c = kidx / TRS, trs = kidx - c * TRS;
                const int ft = trs / RS, rs = trs - ft * RS;
                const int fr = rs / g.S, fs = rs - fr * g.S;
                tab_c[threadIdx.x] = c * (BPROP ? g.M * g.P * g.Q : g.D * g.H * g.W) * g.N;
                tab_d[threadIdx.x] = ft * g.dil_d;
                tab_h[threadIdx.x] = fr * g.dil_h;
                tab_w[threadIdx.x] = fs * g.dil_w;
            } else {
                tab_c[threadIdx.x] = -1;
            }
        }
        __syncthreads();
        for (int i = ty; i < CK; i += 8) {
            T v = 0;
            const int tc = tab_c[i];
            if (tc >= 0 && rvalid) {
                if (BPROP) {
                    const int th = h0 - tab_h[i], tw = w0 - tab_w[i], td = d0 - tab_d[i];
                    if (th >= 0 && tw >= 0 && td >= 0 && th % g.str_h == 0 && tw % g.str_w == 0 &&
                        td % g.str_d == 0) {
                        const int pp = th / g.str_h, q = tw / g.str_w, mm = td / g.str_d;
                        if (pp < g.P && q < g.Q && mm < g.M)
                            v = I[(long long)tc + (((long long)mm * g.P + pp) * g.Q + q) * g.N + n];
                    }
                } else {
                    const int h = h0 + tab_h[i], w = w0 + tab_w[i], dd = d0 + tab_d[i];
                    if (h >= 0 && h < g.H && w >= 0 && w < g.W && dd >= 0 && dd < g.D)
                        v = I[(long long)tc + (((long long)dd * g.H + h) * g.W + w) * g.N + n];
                }
            }
            tile[i][tx] = v;
        }
        __syncthreads();
        if (orow < rows_p) {
            if (MODE == MODE_FLEX16) {
                unsigned hi[4] = {0, 0, 0, 0}, lo[4] = {0, 0, 0, 0};
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int m = (int)tile[vec * 16 + j][wr];
                    const int l = m & 0xff;
                    const int h8 = ((m - l) >> 8) & 0xff;
                    hi[j >> 2] |= (unsigned)h8 << (8 * (j & 3));
                    lo[j >> 2] |= (unsigned)l << (8 * (j & 3));
                }
                const long long o = (long long)orow * kp + kc + vec * 16;
                *reinterpret_cast<uint4*>((unsigned char*)plane0 + o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>((unsigned char*)plane1 + o) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            } else {
                float hi[4], lo[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float a = (float)tile[vec * 4 + j][wr];
                    unsigned hb;
                    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hb) : "f"(a));
                    hi[j] = __uint_as_float(hb);
                    lo[j] = a - hi[j];
                }
                const long long o = (long long)orow * kp + kc + vec * 4;
                *reinterpret_cast<float4*>((float*)plane0 + o) = make_float4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<float4*>((float*)plane1 + o) = make_float4(lo[0], lo[1], lo[2], lo[3]);
            }
        }
    }
}

// ================================================================================================
// Implicit GEMM (flex16): no unrolled copy of the input.
//
// The tile kernel reads the activations straight from their C,H,W,N layout, rows of images padded to 16
// bytes (any batch; images beyond it are zero fill).  A tile is 1x1 to 2x2 output pixels x 128 images;
// its reduction runs over chunks of `cu` input channels.  For every chunk ONE 4-d TMA box [cu channels]
// [window][128 images] per operand plane is fetched: the window under all pixels of the tile in a single
// copy, zero fill outside the image doing the padding.  It lands in shared memory as an MN-major (images
// contiguous) 128-byte-swizzled operand whose K rows are in (channel, row, column of the window) order,
// padded to a multiple of 32 rows (one MMA step).  Each pixel has columns of its own, whose filters stand
// at its place in the window and are zero elsewhere.
//
// At 16..64 output channels an MMA's time is the read of its A operand from shared memory (4 KB
// per instruction whatever N is), so the four byte products are folded into TWO instructions per
// k-step.  The filters' low plane is stored as the signed byte bl - 128, which makes both filter
// planes signed and lets them lie behind one another as one operand of 2*bn rows:
//     A_hi x [B_hi | B_lo'] -> HH | X            A_lo x [B_hi | B_lo'] -> X | LL
// The bias costs 128 * (sum of the activations under the window); that sum comes out of the same
// instructions through one extra filter column whose planes are (0, +1) on every K row: its X and
// LL accumulators are sum(a_hi) and sum(a_lo).  Because that column is 1 on the padding rows too,
// whatever bytes lie there cancel exactly (their true filter value is 0 = 256*0 + (-128) + 128).
//
// The filter planes of the CTA's output channels are loaded ONCE per CTA and stay resident in
// shared memory.  CTAs are persistent: each walks many tiles, the producer warp runs ahead across
// tile boundaries through a ring of stages, and up to four accumulator sets in tensor memory let
// the epilogues of earlier tiles (sixteen warps) overlap the MMAs of later ones.
// The only pre-pass is an elementwise split of the activations into the two operand planes, and a
// fused elementwise kernel that produces the activations can write the planes itself.
// ================================================================================================
struct ConvTileParams {
    int P, Q, N, K;
    int off_h, off_w, step_h, step_w;   // a tile's window starts at tile * step + off
    int cu;                       // channels per chunk
    int cchunks;                  // chunks per tile = stages per tile
    int kc_pad;                   // K rows per chunk, padded to a multiple of 32
    int box_bytes;                // bytes one activation box delivers (cu * window * 128)
    int gh, gw, gw_log, tq;       // output pixels a tile covers (gh x gw), tiles along a row
    int npanels;                  // 128-byte K panels of the resident filter planes
    int nstages;                  // ring depth
    int bn;                       // columns per accumulator: gh*gw * (kt channels + a sum column)
    int kt;                       // output channels per CTA column (blockIdx.y)
    int nbuf;                     // accumulator sets in tensor memory: 1, 2, 3 (or 4)
    int n_mma;                    // MMA-issuing threads: 1..3, at most nbuf
    int tmem_cols;                // power of two >= 3*bn*nbuf
    int num_tiles, nblk;
    long long ldc;
    void* O;
    const b2_flex_scale* table;
    int slotA, slotB, slotC;
    int* stats;
    unsigned long long* probe_out;
    int* status;
    int probe;
    // fused epilogue (all optional): y = relu?(conv + bias[k] + residual) in fp32, quantised once
    // with the output's exponent; stored as int16 and / or as the byte planes the next
    // convolution reads
    const short* bias; int slot_bias;
    const short* residual; int slot_res;      // same K,P,Q,N layout as the output
    const short* mask;                        // likewise: y = mask > 0 ? y : 0
    int relu;
    int write_i16;
    int vec;                      // int16 tensors aligned for eight images at a time
    int NP;                       // images per row of the byte planes
    long long ldc_planes;
    unsigned char* out_planes; long long out_plane_bytes;
};

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int c0, int c1,
                                            int c2, int c3, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
}
// two fp32 values in one 64-bit register, and the packed arithmetic on them
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// eight consecutive int16, as one load where the alignment allows it; only the first n exist
__device__ __forceinline__ uint4 load8(const short* p, int vec, int n) {
    if (n <= 0) return make_uint4(0, 0, 0, 0);
    if (vec) return *reinterpret_cast<const uint4*>(p);
    const unsigned short* q = reinterpret_cast<const unsigned short*>(p);
    unsigned v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = j < n ? q[j] : 0;
    return make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
}
// two values in a word, saturated to int16
__device__ __forceinline__ unsigned pack_sat(int lo, int hi) {
    unsigned r;
    asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(r) : "r"(hi), "r"(lo));
    return r;
}
// bits of the halves of m that are positive
__device__ __forceinline__ unsigned positive2(unsigned m) { return __vmins2(__vmaxs2(m, 0u), 0x00010001u) * 0xffffu; }
// four 8x8 matrices of 16-bit values, rows at each thread's address, transposed
__device__ __forceinline__ uint4 load_turned(const void* row) {
    uint4 r;
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(smem_u32(row)) : "memory");
    return r;
}
// one 32-bit column of this thread's TMEM lane
__device__ __forceinline__ unsigned tmem_ld1(unsigned taddr) {
    unsigned r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(taddr) : "memory");
    return r;
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap* m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}
// instruction descriptor with a run-time N
__device__ __forceinline__ unsigned make_idesc_n(unsigned dfmt, unsigned afmt, unsigned bfmt,
                                                 unsigned n) {
    return (dfmt << 4) | (afmt << 7) | (bfmt << 10) | ((n >> 3) << 17) |
           ((unsigned)(kBlockM >> 4) << 24);
}

constexpr int kConvMaxStages = 8;
constexpr int kConvThreads = 640;           // producer, MMA, sixteen epilogue warps, two more MMA warps
constexpr int kConvSmemMax = 232448;        // 227 KB: the most one CTA can have
constexpr int kConvSmemFixed = 1024 /*alignment*/ + 1024 /*barriers, bias*/ + 16 * 1024 /*epilogue staging*/;

// OFF: 32-bit element offsets into the output where they reach, 64-bit ones for larger tensors.
// EPI: 0 plain integer rescale, 1 fused tail, 2 fused tail with a residual.  MASK: the result is kept
// where another tensor is positive (the gradient of a ReLU).  SHORT: 256*HH + X fits 32 bits.  EVEN: eight images and eight channels at a time throughout -- aligned tensors, channel
// counts that are multiples of eight -- and not a measuring launch.  (Template parameters because a tested-and-skipped block of the epilogue is not free: the
// compiler predicates it, and its instructions are issued all the same -- 60 of 330 per piece.)
enum { EPI_INT = 0, EPI_FUSED = 1, EPI_RESIDUAL = 2 };
template <typename OFF, int EPI, bool SHORT, bool EVEN, bool MASK>
__global__ void __launch_bounds__(kConvThreads, 1)
conv_implicit_kernel(const __grid_constant__ CUtensorMap mapI0,
                     const __grid_constant__ CUtensorMap mapI1,
                     const __grid_constant__ CUtensorMap mapB, const ConvTileParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int bn = p.bn;
    const int panel_bytes = 2 * bn * kKBytes;                  // [B_hi rows | B_lo' rows] x 128 B
    const int acc_cols = 3 * bn;                               // HH | X | LL
    const int act_stage = p.kc_pad * 128;                      // bytes per plane per stage
    unsigned char* filt = smem;                                // [npanels][2*bn][128]
    unsigned char* ring = smem + p.npanels * panel_bytes;      // [nstages][2 planes][act_stage]
    // one set of "stage filled" barriers per MMA-issuing warp: a waiter must see every phase of
    // a barrier in turn (a parity wait cannot tell phase n from phase n+2), and an issuer only
    // ever looks at the stages of its own tiles
    unsigned long long* full_bar =
        (unsigned long long*)(ring + (size_t)p.nstages * 2 * act_stage);   // [4][kConvMaxStages]
    unsigned long long* empty_bar = full_bar + 4 * kConvMaxStages;
    unsigned long long* tmem_full = empty_bar + kConvMaxStages;   // [4]
    // "set drained" barriers, one per (issuing thread, set): the epilogue signals the thread that
    // will fill the set next, so each thread meets every phase of its own barriers in turn
    unsigned long long* tmem_empty = tmem_full + 4;               // [4 issuers][4 sets]
    unsigned long long* filt_bar = tmem_empty + 16;
    unsigned* tmem_holder = (unsigned*)(filt_bar + 1);
    int* fail_flag = (int*)(tmem_holder + 1);
    // [bn] bias of this CTA's channels in units of the output's step; then the epilogue's staging
    float* bias_s = (float*)((unsigned char*)full_bar + 512);
    unsigned char* epi_smem = (unsigned char*)full_bar + 1024;    // 1 KB per epilogue warp

    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int epi_w = p.nbuf == 3 ? 1 : 4 / p.nbuf;   // epilogue warps per lane quarter and accumulator set

    if (threadIdx.x == 0) {
        prefetch_map(&mapI0); prefetch_map(&mapI1); prefetch_map(&mapB);
        for (int s = 0; s < kConvMaxStages; ++s) {
            for (int i = 0; i < 4; ++i) mbar_init(&full_bar[i * kConvMaxStages + s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 4; ++b) {
            mbar_init(&tmem_full[b], 1);
            for (int i = 0; i < 4; ++i) mbar_init(&tmem_empty[i * 4 + b], 4 * epi_w);
        }
        mbar_init(filt_bar, 1);
        *fail_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(tmem_holder, p.tmem_cols);
        // Programmatic dependent launch: the next kernel of the stream, if it was launched the same
        // way, may take the SMs this grid leaves while its last CTAs still work, and do its set-up;
        // it reads and writes global memory only after its own griddepcontrol.wait below.  (Not
        // before this CTA holds its tensor memory, or the two could each wait for what the other has.)
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    // everything before this line touches no global memory; everything after it sees the
    // completed work of all earlier kernels of the stream
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (threadIdx.x >= 64 && threadIdx.x < 64 + bn) {
        const int col = blockIdx.y * p.kt + (int)(threadIdx.x - 64) % p.kt;
        bias_s[threadIdx.x - 64] = (EPI != EPI_INT && p.bias && (int)(threadIdx.x - 64) < p.gh * p.gw * p.kt && col < p.K)
                                       ? (float)p.bias[col] * p.table[p.slot_bias].scale *
                                             (p.probe ? 1.0f : p.table[p.slotC].inv_scale)
                                       : 0.0f;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = (unsigned)warp_uniform((int)*tmem_holder);

    if (warp == 0) {
        if (elect_one()) {
            // the filter planes of this CTA's output channels: once, resident
            mbar_expect_tx(filt_bar, p.npanels * panel_bytes);
            for (int j = 0; j < p.npanels; ++j)
                tma_load_2d(filt + j * panel_bytes, &mapB, j * kKBytes, blockIdx.y * 2 * bn, filt_bar);
            // Every role of this kernel is a single chain of instructions per tile, so nothing in
            // the loops divides: the tile's image block, column and row advance by the fixed step
            // of gridDim.x tiles with carries, and ring positions are counters (the divisions
            // alone cost this thread more than the copies of a small tile take).
            int s = 0, mma = 0;
            const int n_mma = p.n_mma;
            unsigned empty_parity = 1;         // the first pass over the ring finds every stage free
            bool ok = true;
            const int tq = p.tq, nblk = p.nblk;
            int nb = (int)blockIdx.x % nblk, pq = (int)blockIdx.x / nblk, q = pq % tq, pp = pq / tq;
            const int d_nb = (int)gridDim.x % nblk, d_pq = (int)gridDim.x / nblk, d_q = d_pq % tq,
                      d_p = d_pq / tq;
            const int step_h = p.step_h, step_w = p.step_w;
            for (int tile = blockIdx.x; tile < p.num_tiles && ok; tile += gridDim.x) {
                unsigned long long* fb = full_bar + mma * kConvMaxStages;            // its consumer's
                if (++mma == n_mma) mma = 0;
                const int n0 = nb * 128;
                const int h0 = pp * step_h + p.off_h, w0 = q * step_w + p.off_w;
                for (int cc = 0; cc < p.cchunks; ++cc) {
                    if (!mbar_wait(&empty_bar[s], empty_parity)) {
                        atomicExch(fail_flag, 1); ok = false; break;
                    }
                    unsigned char* sa = ring + (size_t)s * 2 * act_stage;
                    mbar_expect_tx(&fb[s], 2 * p.box_bytes);
                    tma_load_4d(sa, &mapI0, n0, w0, h0, cc * p.cu, &fb[s]);
                    tma_load_4d(sa + act_stage, &mapI1, n0, w0, h0, cc * p.cu, &fb[s]);
                    if (++s == p.nstages) { s = 0; empty_parity ^= 1u; }
                }
                nb += d_nb; q += d_q; pp += d_p;
                if (nb >= nblk) { nb -= nblk; ++q; }
                if (q >= tq) { q -= tq; ++pp; }
            }
        }
    } else if (warp == 1 || warp >= 18) {
        // up to three MMA-issuing threads take the tiles in turn (when there are accumulator sets
        // for them), so that the waits of one tile's chunks overlap the next tile's instructions.
        // The issuing thread is picked with elect.sync: under `lane == 0` the compiler cannot
        // see that one thread runs and wraps every instruction in a loop over the active threads
        // (22 launches of a batch-256 pass 364 -> 328 us, the update kernel 622 -> 471 us).
        const int mma_id = warp == 1 ? 0 : warp - 17;
        const int n_mma = p.n_mma;
        if (elect_one()) {
            // bit 15: A is MN-major.  A_hi is signed, A_lo unsigned, both filter planes signed.
            const unsigned mn = 1u << 15;
            const unsigned id_s2 = make_idesc_n(2, 1, 1, 2 * bn) | mn, id_u2 = make_idesc_n(2, 0, 1, 2 * bn) | mn;
            const unsigned id_s1 = make_idesc_n(2, 1, 1, bn) | mn, id_u1 = make_idesc_n(2, 0, 1, bn) | mn;
            bool ok = mma_id < n_mma && mbar_wait(filt_bar, 0);
            if (!ok && mma_id < n_mma) atomicExch(fail_flag, 1);
            const int ksteps = p.kc_pad >> 5;
            // Matrix descriptors as (low word, constant high word): only the start address
            // (bits 0-13, in 16-byte units) changes from one MMA to the next, so the loop keeps
            // a few running integers instead of rebuilding 64-bit descriptors.
            const unsigned long long desc_hi = (unsigned long long)((1024u >> 4) | (1u << 14) | (2u << 29)) << 32;
            const unsigned filt_lo = ((smem_u32(filt) >> 4) & 0x3FFF) | (1u << 16);     // K-major: LBO field 1
            const unsigned lo_rows = (unsigned)((bn * kKBytes) >> 4);                   // B_lo' behind B_hi
            const unsigned panel_units = (unsigned)(panel_bytes >> 4);
            const unsigned ring_lo = (smem_u32(ring) >> 4) & 0x3FFF;                  // MN-major: LBO field 0
            const unsigned stage_units = (unsigned)((2 * act_stage) >> 4), plane_units = (unsigned)(act_stage >> 4);
            int s = 0;
            unsigned phase_bits = 0, stage_lo = ring_lo;       // bit s: parity of my next phase of stage s
            unsigned empty_bits = 0;                           // bit b: the same for set b's "drained" barrier
            unsigned long long* fb = full_bar + mma_id * kConvMaxStages;
            int turn = 0, buf = -1;
            bool first_use = true;                             // the sets start out empty
            for (int tile = blockIdx.x; tile < p.num_tiles && ok; tile += gridDim.x) {
                if (++buf == p.nbuf) { buf = 0; first_use = false; }
                const bool my_turn = turn == mma_id;
                if (++turn == n_mma) turn = 0;
                if (!my_turn) {
                    // the other issuing thread's tile: step over its stages (their "filled"
                    // barriers are the other thread's own)
                    for (int cc = 0; cc < p.cchunks; ++cc) {
                        stage_lo += stage_units;
                        if (++s == p.nstages) { s = 0; stage_lo = ring_lo; }
                    }
                    continue;
                }
                const unsigned acc_base = tmem_base + buf * acc_cols;
                if (!first_use) {
                    if (!mbar_wait(&tmem_empty[mma_id * 4 + buf], (empty_bits >> buf) & 1u)) {
                        atomicExch(fail_flag, 1); ok = false; break;
                    }
                    empty_bits ^= 1u << buf;
                }
                tc_fence_after();
                int idx = 0;                                   // 32-byte column block of the filter planes
                for (int cc = 0; cc < p.cchunks; ++cc) {
                    if (!mbar_wait(&fb[s], (phase_bits >> s) & 1u)) {
                        atomicExch(fail_flag, 1); ok = false; break;
                    }
                    phase_bits ^= 1u << s;
                    tc_fence_after();
                    unsigned a_lo = stage_lo;
                    for (int k = 0; k < ksteps; ++k, ++idx, a_lo += 256u) {
                        const unsigned boff = (unsigned)(idx >> 2) * panel_units + (unsigned)(idx & 3) * 2u;
                        const unsigned long long dB = desc_hi | (filt_lo + boff);
                        const unsigned long long dA0 = desc_hi | a_lo;
                        const unsigned long long dA1 = desc_hi | (a_lo + plane_units);
                        if (idx > 0) {
                            tc_mma<MODE_FLEX16>(acc_base, dA0, dB, id_s2, 1u);            // HH | X
                            tc_mma<MODE_FLEX16>(acc_base + bn, dA1, dB, id_u2, 1u);       // X | LL
                        } else {
                            // first k-step of a tile: the accumulators start from different products
                            const unsigned long long dBl = desc_hi | (filt_lo + boff + lo_rows);
                            tc_mma<MODE_FLEX16>(acc_base, dA0, dB, id_s1, 0u);
                            tc_mma<MODE_FLEX16>(acc_base + bn, dA0, dBl, id_s1, 0u);
                            tc_mma<MODE_FLEX16>(acc_base + bn, dA1, dB, id_u1, 1u);
                            tc_mma<MODE_FLEX16>(acc_base + 2 * bn, dA1, dBl, id_u1, 0u);
                        }
                    }
                    tc_commit(&empty_bar[s]);
                    stage_lo += stage_units;
                    if (++s == p.nstages) { s = 0; stage_lo = ring_lo; }
                }
                tc_commit(&tmem_full[buf]);
            }
        }
    } else {
        // epilogue warps 2..17: TMEM lane quarter = warp % 4.  Accumulator set b is drained by the
        // warps whose slot (0..3) falls into [b*epi_w, (b+1)*epi_w); they take the 16-column
        // chunks of its output channels in turn.
        const int quarter = warp & 3;
        const int slot = (warp - 2) >> 2;
        const int set = slot / epi_w, part = slot % epi_w;
        const int ncol0 = blockIdx.y * p.kt;                  // first output channel of this CTA
        // columns of the accumulators: gh*gw pixels x kt channels, then one sum column per pixel.
        // (a tile of several pixels has kt a multiple of 16, so no piece of columns straddles two
        // pixels; kt > channels left only where K is cut into CTA columns, and then G is 1)
        const int G = p.gh * p.gw, kt = p.kt, ncols = G * kt;
        const int left = p.K - ncol0 < kt ? p.K - ncol0 : kt;  // output channels this CTA owns
        int stat = 0;
        unsigned long long pmax = 0;
        const int n_mma_e = p.n_mma;
        const int n_my = (p.num_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
        const float f = p.table[p.slotA].scale * p.table[p.slotB].scale *
                        (p.probe ? 1.0f : p.table[p.slotC].inv_scale);
        const int sh = -ilogbf(f);
        // fused epilogue: every term carries the output's 1/step (a power of two, so the scaled
        // sum is the real-valued sum times that power, bit for bit); the probe keeps real values
        const float q_out = p.probe ? 1.0f : p.table[p.slotC].inv_scale;
        const float f_conv = p.table[p.slotA].scale * p.table[p.slotB].scale * q_out;
        const float s_res = EPI == EPI_RESIDUAL ? p.table[p.slot_res].scale * q_out : 0.0f;
        const unsigned long long s_res2 = pack2(s_res, s_res), f_conv2 = pack2(f_conv, f_conv),
                                 k256 = pack2(256.0f, 256.0f), k65536 = pack2(65536.0f, 65536.0f);
        float fstat = 0.0f;
        const OFF ldc = (OFF)p.ldc, ldc_p = (OFF)p.ldc_planes;
        unsigned char* const out_lo = p.out_planes + p.out_plane_bytes;
        const bool fast = sh >= 1 && sh <= 31;
        const unsigned rmask = fast ? (1u << sh) - 1u : 0u, rhalf = fast ? 1u << (sh - 1) : 0u;
        bool ok = true;
        // this warp's tiles: every nbuf-th one of the CTA; `next` is the issuing thread of the
        // tile that follows in the same accumulator set.  Coordinates advance with carries, as in
        // the producer.
        const int buf = set, nbuf = p.nbuf, d_next = nbuf % n_mma_e;
        int next = (set + nbuf) % n_mma_e;
        unsigned full_parity = 0;
        const int tq = p.tq, nblk = p.nblk;
        const int first = (int)blockIdx.x + set * (int)gridDim.x, step = nbuf * (int)gridDim.x;
        int nb = first % nblk, pq = first / nblk, tx = pq % tq, ty = pq / tq;
        const int d_nb = step % nblk, d_pq = step / nblk, d_x = d_pq % tq, d_y = d_pq / tq;
        // Stores and the residual go through 512 bytes of shared memory of this warp each: a
        // thread computes one image of eight channels, but stores eight images of one channel --
        // one 8-byte store per plane (16 bytes for int16) in place of eight of one byte.
        // Two halves used in turn, so that one __syncwarp between writing and reading is enough.
        unsigned char* const stage_smem = epi_smem + (warp - 2) * 1024;
        unsigned stage = 0;
        const int epi_mask = epi_w - 1, kt8 = (kt + 7) >> 3 & epi_mask;
        // plain rescale in 32-bit pieces: where the sums fit and the shift takes at least the low byte
        const bool exact32 = EPI == EPI_INT && SHORT && !p.probe && sh >= 9 && sh <= 38;
        const unsigned rmask8 = exact32 ? (1u << (sh - 8)) - 1u : 0u, rhalf8 = exact32 ? 1u << (sh - 9) : 0u;
        unsigned smx = 0, smn = 0;                             // packed pairs: largest and smallest mantissa
        const bool probing = !EVEN && p.probe;
        const float z_lo = p.relu ? 0.0f : (probing ? -INFINITY : -32768.0f),
                    z_hi = probing ? INFINITY : 32767.0f;
        const int scol = lane >> 2;                            // channel of the piece this lane stores
        const int simg = quarter * 32 + (lane & 3) * 8;        // and its first image in the tile
        // A thread's eight channels of an image are 16 bytes, a row of the 8x8 matrices that ldmatrix turns round.  Rows are
        // dealt to the matrices so that a thread gets eight images in order, and stored where the rows of a matrix lie in
        // eight different banks.  (Instruction issue: with a 16-bit store for every value, clamps before a magic-number add
        // and a comparison for the mask a step of ResNet-20 in training, batch 1024, spent 1135 us here, 1083 so; layers
        // with a residual 47.5 -> 42 us.)
        const unsigned floor2 = p.relu ? 0u : 0x80008000u;
        const int turn_to = ((lane & ~7) | ((lane + 2 * (lane >> 3)) & 7)) * 16;
        const int turn_from = (8 * ((lane & 7) >> 1) + ((2 * (lane >> 3) + (lane & 1) + 2 * ((lane & 7) >> 1)) & 7)) * 16;
        // (with three sets the warps of the fourth slot have none)
        for (int ti = set < nbuf ? set : n_my; ti < n_my; ti += nbuf) {
            const int p0 = ty * p.gh, q0 = tx * p.gw;
            // a pixel of the tile: inside the image or not, and its offset within a channel (of the
            // int16 tensors; the planes' where their rows are padded)
            OFF poff = 0;
            auto pixel = [&](int g, OFF& off) -> bool {
                const int gy = g >> p.gw_log, gx = g & (p.gw - 1);
                const OFF pix = (OFF)((p0 + gy) * p.Q + q0 + gx);
                off = pix * (OFF)p.N + (OFF)(nb * 128);
                if (!EVEN) poff = pix * (OFF)p.NP + (OFF)(nb * 128);
                return p0 + gy < p.P && q0 + gx < p.Q;
            };
            // images beyond N in the last block of a ragged batch: this thread's own, and how many of
            // the eight that it loads and stores exist
            const bool live_img = EVEN || nb * 128 + quarter * 32 + lane < p.N;
            const int n_img = EVEN ? 8 : p.N - (nb * 128 + simg);
            if (EPI != EPI_INT || exact32) {
                // Eight columns at a time, loads first, then arithmetic, then stores: eight independent
                // chains.  The warps that share a lane quarter take the 8-column pieces in turn.
                //   fused: the exact integer sum scaled to a real value in fp32, bias and residual added,
                //   ReLU, ONE quantisation with the output's exponent; sums two at a time (fma.f32x2);
                //   plain: the exact sum in 32-bit halves, rescaled with round to nearest even.
                // Instruction issue bounds it, so choices are made once per pixel or piece, addresses
                // once per pixel, and the statistic is taken on packed pairs.
                uint4 rq = make_uint4(0, 0, 0, 0), mq = make_uint4(0, 0, 0, 0);
                // residual and mask of a piece, fetched one piece ahead of its use
                auto fetch = [&](OFF at) {
                    if (EPI == EPI_RESIDUAL) rq = load8(p.residual + at, EVEN || p.vec, n_img);
                    if (MASK) mq = load8(p.mask + at, EVEN || p.vec, n_img);
                };
                constexpr bool AHEAD = EPI == EPI_RESIDUAL || MASK;
                OFF off;
                bool inside = pixel(0, off);
                off += (OFF)(ncol0 + scol) * ldc + (OFF)simg;
                int c = (part & epi_mask) * 8;
                if (AHEAD && inside && c < kt && (EVEN || c + scol < left)) fetch(off + (OFF)c * ldc);
                if (ok && !mbar_wait(&tmem_full[buf], full_parity)) { atomicExch(fail_flag, 1); ok = false; }
                tc_fence_after();
                const unsigned lane_addr = tmem_base + buf * acc_cols + ((unsigned)(quarter * 32) << 16);
                bool ahead = false;
                for (int g = 0, start = part; g < G; ++g) {
                    // 128 * (sum of the activations under the pixel's window), from its sum column
                    // (|sum of activations| < 2^30: exact in 32 bits)
                    const unsigned s_hi = tmem_ld1(lane_addr + bn + ncols + g);
                    const unsigned s_lo = tmem_ld1(lane_addr + 2 * bn + ncols + g);
                    tmem_ld_wait();
                    const int act_sum = (int)(s_hi * 256u + s_lo);
                    const float fixf = 128.0f * (float)act_sum;
                    const unsigned long long fix2 = pack2(fixf, fixf);
                    const unsigned col0 = lane_addr + g * kt;
                    const bool here = inside && ok;
                    const OFF at_g = off, poff_g = poff + (OFF)(ncol0 + scol) * ldc_p + (OFF)simg;
                    start = (start + epi_w - kt8) & epi_mask;     // first piece of this warp in pixel g+1
                    for (; c < kt; c += 8 * epi_w) {
                        unsigned hh[8], xx[8], ll[8];
                        tmem_ld8(col0 + c, hh);
                        tmem_ld8(col0 + bn + c, xx);
                        tmem_ld8(col0 + 2 * bn + c, ll);
                        const int live = left - c;
                        const OFF at = at_g + (OFF)c * ldc;
                        unsigned long long y[4];
                        if (EPI != EPI_INT) {
                            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(bias_s + c);
                            const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(bias_s + c + 4);
                            y[0] = b0.x; y[1] = b0.y; y[2] = b1.x; y[3] = b1.y;
                        }
                        const uint4 m_now = mq;
                        stage ^= 512;
                        if (EPI == EPI_RESIDUAL) {
                            *reinterpret_cast<uint4*>(stage_smem + stage + lane * 16) = rq;
                            __syncwarp();
                            const short* rs = reinterpret_cast<const short*>(stage_smem + stage + lane * 2);
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                y[j] = fma2(pack2((float)rs[64 * j], (float)rs[64 * j + 32]), s_res2, y[j]);
                            stage ^= 512;
                        }
                        if (AHEAD) {
                            int cn = c + 8 * epi_w;
                            OFF offn = at_g;
                            const OFF keep = poff;
                            bool in = inside;
                            if (cn >= kt && g + 1 < G) {
                                in = pixel(g + 1, offn);
                                offn += (OFF)(ncol0 + scol) * ldc + (OFF)simg;
                                cn = start * 8;
                                ahead = true;
                            }
                            poff = keep;
                            if (in && cn < kt && (EVEN || cn + scol < left)) fetch(offn + (OFF)cn * ldc);
                        }
                        tmem_ld_wait();
                        if (!here) continue;
                        unsigned short* so = reinterpret_cast<unsigned short*>(stage_smem + stage + lane * 2);
                        unsigned pk[4];
                        if (EPI == EPI_INT) {
                            // w = floor(sum / 256), r = sum mod 256; q = w / 2^(sh-8) to nearest, ties
                            // (r = 0) to even
                            const int fix = 128 * act_sum;
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const int l = (int)ll[j] + fix, w = (int)(hh[j] << 8) + (int)xx[j] + (l >> 8);
                                const unsigned rem = (unsigned)w & rmask8;
                                int q = w >> (sh - 8);
                                const unsigned odd = (unsigned)q & 1u;
                                q += (rem > rhalf8 || (rem == rhalf8 && (odd | ((unsigned)l & 255u)))) ? 1 : 0;
                                hh[j] = (unsigned)q;
                            }
#pragma unroll
                            for (int j = 0; j < 4; ++j) pk[j] = pack_sat((int)hh[2 * j], (int)hh[2 * j + 1]);
                        } else {
                            if (SHORT) {
                                // 256*HH + X fits 32 bits: two conversions a value instead of three
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    const unsigned long long t =
                                        pack2((float)(int)((hh[2 * j] << 8) + xx[2 * j]),
                                              (float)(int)((hh[2 * j + 1] << 8) + xx[2 * j + 1]));
                                    const unsigned long long l =
                                        add2(pack2((float)(int)ll[2 * j], (float)(int)ll[2 * j + 1]), fix2);
                                    y[j] = fma2(fma2(t, k256, l), f_conv2, y[j]);
                                }
                            } else {
                                // correctly rounded conversions instead of a 64-bit sum: the fp32
                                // result is quantised to 16 bits right after
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    const unsigned long long l =
                                        add2(pack2((float)(int)ll[2 * j], (float)(int)ll[2 * j + 1]), fix2);
                                    const unsigned long long x =
                                        fma2(pack2((float)(int)xx[2 * j], (float)(int)xx[2 * j + 1]), k256, l);
                                    const unsigned long long h = pack2((float)(int)hh[2 * j], (float)(int)hh[2 * j + 1]);
                                    y[j] = fma2(fma2(h, k65536, x), f_conv2, y[j]);
                                }
                            }
                            if (!EVEN && p.probe) {
                                // the largest |value| (kept where the mask is positive)
                                float z[8];
#pragma unroll
                                for (int j = 0; j < 4; ++j) unpack2(y[j], z[2 * j], z[2 * j + 1]);
#pragma unroll
                                for (int j = 0; j < 8; ++j) z[j] = fminf(fmaxf(z[j], z_lo), z_hi);
                                if (MASK) {
                                    *reinterpret_cast<uint4*>(stage_smem + stage + lane * 16) = m_now;
                                    __syncwarp();
#pragma unroll
                                    for (int j = 0; j < 8; ++j) z[j] = (short)so[32 * j] > 0 ? z[j] : 0.0f;
                                }
#pragma unroll
                                for (int j = 0; j < 8; ++j)
                                    if (j < live && live_img) fstat = fmaxf(fstat, fabsf(z[j]));
                                __syncwarp();
                                continue;
                            }
                            // in units of the output's step (see f_conv): rounded to nearest even and saturated by the
                            // conversions, ReLU on pairs.  (No NaN can arise: every term is finite.)
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                float a, b;
                                unpack2(y[j], a, b);
                                pk[j] = __vmaxs2(pack_sat(__float2int_rn(a), __float2int_rn(b)), floor2);
                            }
                        }
                        *reinterpret_cast<uint4*>(stage_smem + stage + turn_to) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                        __syncwarp();
                        uint4 w = load_turned(stage_smem + stage + turn_from);
                        if (MASK) {
                            w.x &= positive2(m_now.x); w.y &= positive2(m_now.y);
                            w.z &= positive2(m_now.z); w.w &= positive2(m_now.w);
                        }
                        if (EVEN || (scol < live && n_img > 0)) {
                            if (!EVEN && n_img < 8) {
                                // images beyond the batch count for nothing
                                unsigned* v = reinterpret_cast<unsigned*>(&w);
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                    v[j] &= (2 * j < n_img ? 0xffffu : 0u) | (2 * j + 1 < n_img ? 0xffff0000u : 0u);
                            }
                            smx = __vimax3_s16x2(__vimax3_s16x2(smx, w.x, w.y), w.z, w.w);
                            smn = __vimin3_s16x2(__vimin3_s16x2(smn, w.x, w.y), w.z, w.w);
                            if (EPI != EPI_INT && p.out_planes) {
                                // (rows of the planes are padded to 16 images: all eight have a place)
                                const OFF pat = EVEN ? at : poff_g + (OFF)c * ldc_p;
                                *reinterpret_cast<uint2*>(p.out_planes + pat) =
                                    make_uint2(__byte_perm(w.x, w.y, 0x7531), __byte_perm(w.z, w.w, 0x7531));
                                *reinterpret_cast<uint2*>(out_lo + pat) =
                                    make_uint2(__byte_perm(w.x, w.y, 0x6420), __byte_perm(w.z, w.w, 0x6420));
                            }
                            if (EVEN || p.vec) {
                                if (EPI == EPI_INT || p.write_i16) *reinterpret_cast<uint4*>((short*)p.O + at) = w;
                            } else if (EPI == EPI_INT || p.write_i16) {
                                const unsigned v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll 1
                                for (int j = 0; j < 8 && j < n_img; ++j)
                                    ((short*)p.O)[at + j] = (short)((j & 4 ? (j & 2 ? v[3] : v[2])
                                                                           : (j & 2 ? v[1] : v[0])) >> 16 * (j & 1));
                            }
                        }
                    }
                    if (g + 1 < G) {
                        inside = pixel(g + 1, off);
                        off += (OFF)(ncol0 + scol) * ldc + (OFF)simg;
                        c = start * 8;
                        // (a pixel in which this warp had no piece has fetched nothing ahead)
                        if (AHEAD && !ahead && inside && c < kt && (EVEN || c + scol < left))
                            fetch(off + (OFF)c * ldc);
                        ahead = false;
                    }
                }
            } else {
                if (ok && !mbar_wait(&tmem_full[buf], full_parity)) { atomicExch(fail_flag, 1); ok = false; }
                tc_fence_after();
                const unsigned lane_addr = tmem_base + buf * acc_cols + ((unsigned)(quarter * 32) << 16);
                for (int c0 = part * 16; c0 < ncols; c0 += 16 * epi_w) {
                    unsigned hh[16], xx[16], ll[16];
                    const int g = G == 1 ? 0 : c0 / kt, chan = c0 - g * kt;
                    OFF off;
                    const bool inside = pixel(g, off);
                    off += (OFF)(ncol0 + chan) * ldc + (OFF)(quarter * 32 + lane);
                    const unsigned s_hi = tmem_ld1(lane_addr + bn + ncols + g);
                    const unsigned s_lo = tmem_ld1(lane_addr + 2 * bn + ncols + g);
                    tmem_ld16(lane_addr + c0, hh);
                    tmem_ld16(lane_addr + bn + c0, xx);
                    tmem_ld16(lane_addr + 2 * bn + c0, ll);
                    tmem_ld_wait();
                    const int live = left - chan;
                    if (!ok || !inside || !live_img) continue;
                    short* out = (short*)p.O + off;
                    const long long fix = 128LL * (long long)(int)(s_hi * 256u + s_lo);
                    long long v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        v[j] = ((long long)(int)hh[j] << 16) + ((long long)(int)xx[j] << 8) +
                               (long long)(int)ll[j] + fix;
                    if (p.probe) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const unsigned long long a = (unsigned long long)(v[j] < 0 ? -v[j] : v[j]);
                            if (j < live) pmax = a > pmax ? a : pmax;
                        }
                        continue;
                    }
                    // all sixteen values first, then the stores: independent chains for the scheduler
                    int q[16];
                    if (fast) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) q[j] = rescale_i64_fast(v[j], sh, rmask, rhalf);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j) q[j] = rescale_i64(v[j], sh);
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (j < live) {
                            const int a = q[j] < 0 ? -q[j] : q[j];
                            stat = a > stat ? a : stat;
                            out[(long long)j * p.ldc] = (short)q[j];
                        }
                    }
                }
            }
            full_parity ^= 1u;
            nb += d_nb; tx += d_x; ty += d_y;
            if (nb >= nblk) { nb -= nblk; ++tx; }
            if (tx >= tq) { tx -= tq; ++ty; }
            // this warp has read its part of the accumulator set
            tc_fence_before();
            __syncwarp();
            // tell the thread that fills this set next (tile ti + nbuf of this CTA, if there is one)
            if (lane == 0 && ti + nbuf < n_my) mbar_arrive(&tmem_empty[next * 4 + buf]);
            next += d_next;
            if (next >= n_mma_e) next -= n_mma_e;
        }
        if (p.probe) {
            // fused: the bit pattern of max |y| (fp32); plain: max |integer sum|
            if (EPI != EPI_INT) pmax = (unsigned long long)__float_as_uint(fstat);
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long t = __shfl_xor_sync(0xffffffffu, pmax, o);
                pmax = t > pmax ? t : pmax;
            }
            if (lane == 0 && pmax) atomicMax(p.probe_out, pmax);
        } else {
            const int hi = max((int)(short)smx, (int)smx >> 16), lo = min((int)(short)smn, (int)smn >> 16);
            stat = max(stat, max(hi, -lo));
            for (int o = 16; o > 0; o >>= 1) {
                const int t = __shfl_xor_sync(0xffffffffu, stat, o);
                stat = t > stat ? t : stat;
            }
            if (lane == 0 && stat) atomicMax(p.stats + p.slotC, stat);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, p.tmem_cols);
    }
    if (threadIdx.x == 0 && *fail_flag && p.status) atomicExch(p.status, 1);
}

// activations -> two operand planes in the same C,H,W,N layout, eight mantissas per thread: one 16-byte
// load, two 8-byte stores
__global__ void __launch_bounds__(256)
split_same_layout_kernel(const short* __restrict__ src, long long n8, void* __restrict__ plane0,
                         void* __restrict__ plane1) {
    after_earlier_kernels();
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n8; v += stride) {
        const uint4 w = __ldcs(reinterpret_cast<const uint4*>(src) + v);
        reinterpret_cast<uint2*>(plane0)[v] = make_uint2(__byte_perm(w.x, w.y, 0x7531), __byte_perm(w.z, w.w, 0x7531));
        reinterpret_cast<uint2*>(plane1)[v] = make_uint2(__byte_perm(w.x, w.y, 0x6420), __byte_perm(w.z, w.w, 0x6420));
    }
}

// the same into planes whose rows of n images are padded to np
__global__ void __launch_bounds__(256)
split_padded_kernel(const short* __restrict__ src, long long rows, int n, int np,
                    unsigned char* __restrict__ plane0, unsigned char* __restrict__ plane1) {
    after_earlier_kernels();
    const int g8 = np / 8;
    const long long total = rows * g8, stride = (long long)gridDim.x * blockDim.x;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < total; v += stride) {
        const long long row = v / g8;
        const int i0 = (int)(v - row * g8) * 8;
        const unsigned short* q = (const unsigned short*)src + row * n + i0;
        unsigned w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = i0 + j < n ? q[j] : 0u;
        uint2 h, l;
        l.x = (w[0] & 0xff) | (w[1] & 0xff) << 8 | (w[2] & 0xff) << 16 | w[3] << 24;
        l.y = (w[4] & 0xff) | (w[5] & 0xff) << 8 | (w[6] & 0xff) << 16 | w[7] << 24;
        h.x = w[0] >> 8 | (w[1] >> 8) << 8 | (w[2] >> 8) << 16 | (w[3] >> 8) << 24;
        h.y = w[4] >> 8 | (w[5] >> 8) << 8 | (w[6] >> 8) << 16 | (w[7] >> 8) << 24;
        *(uint2*)(plane0 + row * np + i0) = h;
        *(uint2*)(plane1 + row * np + i0) = l;
    }
}

// int16 tensor [c][h][w][n] -> its two byte planes, the low one plane_bytes behind the high one
int split_to_planes(const short* x, int c, int h, int w, int n, void* planes, size_t plane_bytes,
                    cudaStream_t st) {
    const int np = plane_pitch(n);
    const long long rows = (long long)c * h * w, units = rows * np / 8;
    long long blocks = (units + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    unsigned char* lo = (unsigned char*)planes + plane_bytes;
    if (np == n && ((uintptr_t)x & 15) == 0)
        B2_CUDA(b2::launch_after(split_same_layout_kernel, dim3((unsigned)blocks), 256, 0, st, x, units, planes, lo));
    else
        B2_CUDA(b2::launch_after(split_padded_kernel, dim3((unsigned)blocks), 256, 0, st, x, rows, n, np, (unsigned char*)planes, lo));
    B2_CUDA(cudaGetLastError());
    return B2_OK;
}

// filters C,R,S,K -> ONE array [ntn][2*bn rows][kp] for the implicit kernel: for every CTA column
// the high bytes of its output channels (rows 0..bn-1) and, behind them, the low bytes minus 128 as
// signed bytes (rows bn..2bn-1).  A tile covers gh x gw output pixels: row g*kt + k holds output
// channel k as pixel g sees it inside the common window of wh x ww taps (forward: shifted by
// (g/gw)*str_h, (g%gw)*str_w; input gradient: the taps of its own residue modulo the stride, flipped);
// row gh*gw*kt + g is pixel g's sum column: 0 in the high half, +1 in the low half on the taps of its
// own R x S window.  Everything else -- taps of the common window that
// are not the pixel's, channels beyond C, padding -- is zero in both halves, so it adds nothing
// whatever the operand holds there.  The K positions of chunk cc start at cc*kc_pad and run over
// (channel within the chunk, tap row, tap column).
struct FilterLayout {
    int C, R, S, K, cu, cchunks, kc_pad, ntn, bn, kt, kp, gh, gw, str_h, str_w, wh, ww;
    int bprop, off_h, off_w, pad_h, pad_w;
};

// Filters of several convolutions to a launch: a training step rebuilds the planes of every layer, 43
// launches of 2 us for ResNet-20.  A thread makes 16 positions of a row, of both halves: those of a step took 46 us
// when it made one byte and found its place anew for each, 1.2 % of a step at batch 1024 (1933 -> 1910 us with it).
constexpr int kFilterUnit = 16;
constexpr int kFilterJobs = 32;                    // (the argument stays below 4 KB)
struct FilterJobs {
    int n, first[kFilterJobs + 1];                 // job j owns blocks first[j] .. first[j+1]-1
    const short* F[kFilterJobs];
    unsigned char* planes[kFilterJobs];
    FilterLayout layout[kFilterJobs];
};

__global__ void __launch_bounds__(256)
filter_planes_kernel(const __grid_constant__ FilterJobs jobs) {
    after_earlier_kernels();
    int j = 0;
    while (j + 1 < jobs.n && (int)blockIdx.x >= jobs.first[j + 1]) ++j;
    const FilterLayout& f = jobs.layout[j];
    const short* __restrict__ F = jobs.F[j];
    unsigned char* __restrict__ planes = jobs.planes[j];
    const int G = f.gh * f.gw, RS = f.R * f.S, taps = f.wh * f.ww, units = f.kp / kFilterUnit;
    const int total = f.ntn * f.bn * units, stride = (jobs.first[j + 1] - jobs.first[j]) * (int)blockDim.x;
    for (int i = ((int)blockIdx.x - jobs.first[j]) * (int)blockDim.x + threadIdx.x; i < total; i += stride) {
        const int col = i % f.bn, kc = i / f.bn % units * kFilterUnit, tile = i / f.bn / units;
        const int cc = kc / f.kc_pad, within = kc - cc * f.kc_pad;          // (a unit lies in one chunk)
        int cl = within / taps, th = (within - cl * taps) / f.ww, tw = within - cl * taps - th * f.ww;
        const bool sum_col = col >= G * f.kt;
        const int g = sum_col ? col - G * f.kt : col / f.kt, k = tile * f.kt + (sum_col ? 0 : col % f.kt);
        const int gy = g / f.gw, gx = g - gy * f.gw;
        const bool live = g < G && k < f.K && cc < f.cchunks;
        unsigned hi[kFilterUnit / 4], lo[kFilterUnit / 4];
#pragma unroll
        for (int q = 0; q < kFilterUnit; ++q) {
            if (q % 4 == 0) hi[q / 4] = lo[q / 4] = 0;
            const int c = cc * f.cu + cl;
            const int r = f.bprop ? gy + f.pad_h - f.str_h * (f.off_h + th) : th - gy * f.str_h;
            const int s = f.bprop ? gx + f.pad_w - f.str_w * (f.off_w + tw) : tw - gx * f.str_w;
            if (live && r >= 0 && r < f.R && s >= 0 && s < f.S && cl < f.cu && c < f.C) {
                if (sum_col) {
                    lo[q / 4] |= 1u << (8 * (q % 4));
                } else {
                    // bprop: the filter tensor is that of the FORWARD convolution, [K outputs here =
                    // its input channels][R][S][C reduced here = its output channels]
                    const int at = r * f.S + s;
                    const int m = f.bprop ? (int)__ldg(F + ((long long)k * RS + at) * f.C + c)
                                          : (int)__ldg(F + ((long long)c * RS + at) * f.K + k);
                    const int low = m & 0xff;
                    lo[q / 4] |= (unsigned)(low ^ 0x80) << (8 * (q % 4));
                    hi[q / 4] |= (unsigned)(((m - low) >> 8) & 0xff) << (8 * (q % 4));
                }
            }
            if (++tw == f.ww) {
                tw = 0;
                if (++th == f.wh) { th = 0; ++cl; }
            }
        }
        unsigned char* out = planes + ((long long)tile * 2 * f.bn + col) * f.kp + kc;
        *(uint4*)out = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *(uint4*)(out + (long long)f.bn * f.kp) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
}

// int8 plane in C,H,W,N layout; box = [cu][wh][ww][128 images]
int make_map_4d(CUtensorMap* map, void* base, const ConvGeom& g, int cu, int wh, int ww) {
    cuuint64_t dims[4] = {(cuuint64_t)g.N, (cuuint64_t)g.W, (cuuint64_t)g.H, (cuuint64_t)g.C};
    const cuuint64_t np = plane_pitch(g.N);
    cuuint64_t strides[3] = {np, (cuuint64_t)g.W * np, (cuuint64_t)g.H * g.W * np};
    cuuint32_t box[4] = {(cuuint32_t)kKBytes, (cuuint32_t)ww, (cuuint32_t)wh, (cuuint32_t)cu};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, base, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return b2::fail(B2_ERR_CUDA, "cuTensorMapEncodeTiled (4-d) failed (%d)", (int)r);
    return B2_OK;
}

struct ImplicitShape {
    int ntn, kt, bn, nbuf, tmem_cols, cu, cchunks, kc_pad, npanels, kp, nstages, smem;
    int gh, gw, wh, ww, off_h, off_w, step_h, step_w, tiles;
    size_t act_plane, filt_bytes, bytes;
};

// the shape with tiles of gh x gw output pixels; nstages < 2 where it does not fit
ImplicitShape implicit_shape_for(const ConvGeom& g, int gh, int gw) {
    ImplicitShape s;
    s.gh = gh; s.gw = gw;
    window(g.bprop, gh, g.R, g.pad_h, g.str_h, &s.wh, &s.off_h, &s.step_h);
    window(g.bprop, gw, g.S, g.pad_w, g.str_w, &s.ww, &s.off_w, &s.step_w);
    const int G = gh * gw, taps = s.wh * s.ww;
    s.tiles = ((g.P + gh - 1) / gh) * ((g.Q + gw - 1) / gw) * image_blocks(g.N);
    // output channels per CTA column: with the sum columns the two filter planes make one operand
    // of at most 256 rows; in a tile of several pixels a multiple of 16 (no piece of columns
    // straddles two pixels)
    const int most = G == 1 ? 127 : (128 / G - 1) / 16 * 16;
    if (G == 1) {
        s.ntn = (g.K + most - 1) / most;
        s.kt = (g.K + s.ntn - 1) / s.ntn;
    } else {
        s.kt = round_up(g.K, 16) < most ? round_up(g.K, 16) : most;
        s.ntn = (g.K + s.kt - 1) / s.kt;
    }
    s.bn = round_up(G * (s.kt + 1), 16);
    const int sets = 512 / (3 * s.bn);
    s.nbuf = sets >= 4 ? 4 : sets >= 3 ? 3 : sets >= 2 ? 2 : 1;
    s.tmem_cols = 32;
    while (s.tmem_cols < 3 * s.bn * s.nbuf) s.tmem_cols *= 2;
    // channels per chunk: about 36 KB for the two planes of a stage (a 3x3 chunk of 16 channels is
    // 144 rows of 128 bytes), so that several stages are in flight; 1x1 windows take up to 128 channels
    if (taps == 1) s.cu = g.C >= 128 ? 128 : round_up(g.C, 32);
    else s.cu = taps > 64 ? 2 : taps > 20 ? 4 : taps > 10 ? 8 : taps > 4 ? 16 : 32;
    s.cchunks = (g.C + s.cu - 1) / s.cu;
    s.kc_pad = round_up(s.cu * taps, 32);
    s.kp = round_up(s.cchunks * s.kc_pad, kKBytes);
    s.npanels = s.kp / kKBytes;
    const int filt_smem = s.npanels * 2 * s.bn * kKBytes;
    const int stage = 2 * s.kc_pad * 128;
    int nst = (kConvSmemMax - kConvSmemFixed - filt_smem) / stage;
    if (nst > kConvMaxStages) nst = kConvMaxStages;
    s.nstages = s.bn > 128 || s.wh > 256 || s.ww > 256 || s.kt < 1 ? 0 : nst;
    s.smem = kConvSmemFixed + filt_smem + (nst > 0 ? nst : 0) * stage;
    s.act_plane = plane_size(g.C, g.H, g.W, g.N);
    s.filt_bytes = (((size_t)s.ntn * 2 * s.bn * s.kp) + 1023) / 1024 * 1024;
    s.bytes = 2 * s.act_plane + s.filt_bytes;
    return s;
}

// Cycles of a launch with that shape, from the costs measured on the kernel with parts of it taken
// out: an MMA instruction takes the tensor pipe bn cycles (N = 2*bn) but its issuer at least 46;
// the operand fetch runs at 64 bytes a clock and SM; a column costs the sixteen epilogue warps 27;
// and every tile about 300 for the hand-overs between the roles, whatever it holds.
long long implicit_cost(const ImplicitShape& s) {
    const long long mma = (long long)s.cchunks * (s.kc_pad / 32) * 2 * (s.bn > 46 ? s.bn : 46);
    const long long fetch = (long long)s.cchunks * s.cu * s.wh * s.ww * 2 * 128 / 64;
    const long long epi = 27LL * s.gh * s.gw * s.kt;
    long long t = mma > fetch ? mma : fetch;
    if (epi > t) t = epi;
    return (long long)((s.tiles * s.ntn + 147) / 148) * (t + 300);
}

// How many output pixels a tile covers: few channels leave the tensor pipe and the hand-overs
// between the roles mostly idle on one pixel (a 16-channel 3x3 layer spends 550 cycles of a tile on
// twelve narrow instructions and as many on waiting), and neighbouring pixels share most of their
// window.  One pixel where the channels fill the operand, where a group would leave SMs without
// a tile, or where the window grows too much (strides).
//
// The input gradient of a strided convolution needs tiles that are multiples of the stride: then every
// pixel of a tile reads its own residue class of taps from the error tensor as it lies, without the
// zeros that dilating it would put between its elements.
ImplicitShape implicit_shape(const ConvGeom& g) {
    const int sh = g.bprop ? g.str_h : 1, sw = g.bprop ? g.str_w : 1;
    ImplicitShape best = implicit_shape_for(g, sh, sw);
    if (g.K % 16 != 0) return best;
    for (int a = 1; a <= 2; ++a)
        for (int b = 1; b <= 2; ++b) {
            const int gh = sh * a, gw = sw * b;
            if (a * b == 1 || gh * gw > 4 || gw == 3) continue;
            const ImplicitShape s = implicit_shape_for(g, gh, gw);
            if (s.nstages >= 3 && s.bn <= 80 && implicit_cost(s) < implicit_cost(best)) best = s;
        }
    return best;
}

// flex16 only: an MN-major tf32 operand needs the 32-byte-atom variant of the 128-byte swizzle
// (both in the tensor map and in the matrix descriptor); with the plain 128-byte swizzle the
// tensor core reads zeros.  fp32 convolutions therefore gather K-major operands (direct_kernel, or the
// unrolled planes), and so do dilated filters and windows too large for two stages of shared memory.
bool implicit_ok(int mode, const ConvGeom& g) {
    if (mode != MODE_FLEX16 || g.dil_h != 1 || g.dil_w != 1 || getenv("B2_CONV_IM2COL")) return false;
    if (!flat_depth(g)) return false;
    if (g.R > 256 || g.S > 256 || (long long)g.P * g.Q * image_blocks(g.N) >= (1LL << 30)) return false;
    if (g.bprop && (g.str_h * g.str_w > 4 || g.str_w == 3)) return false;
    // the exact int32 sums: |X| <= 2*128*255 per K row
    if ((long long)g.C * g.R * g.S + 32 > 32768) return false;
    return implicit_shape(g).nstages >= 2;
}

// geometry of the implicit kernel for a pass (0 forward, 1 input gradient); false if unsupported.
// The input gradient streams the error tensor (K channels, P x Q) and writes the input's shape.
bool pass_geom(const ConvGeom& f, int pass, ConvGeom* g) {
    *g = f;
    if (pass == 1) {
        g->bprop = 1;
        g->C = f.K; g->H = f.P; g->W = f.Q; g->K = f.C; g->P = f.H; g->Q = f.W;
    }
    return (pass == 0 || pass == 1) && implicit_ok(MODE_FLEX16, *g);
}

// The three parts of an implicit-GEMM convolution: the two operand pre-passes (which a caller can skip
// when it already holds the planes) and the tile kernel.
template <typename T, int MODE>
int implicit_split_activations(const T* I, const ConvGeom& g, const ImplicitShape& s, void* planes,
                               cudaStream_t st) {
    return split_to_planes((const short*)I, g.C, g.H, g.W, g.N, planes, s.act_plane, st);
}

int add_filter_job(FilterJobs* jobs, const void* F, const ConvGeom& g, const ImplicitShape& s, void* planes) {
    const long long n_f = (long long)s.ntn * 2 * s.bn * s.kp;
    B2_REQUIRE(n_f < (1LL << 30), "filter tensor too large");
    long long fb = (n_f / (2 * kFilterUnit) + 255) / 256;
    if (fb > 148 * 8) fb = 148 * 8;
    const int j = jobs->n++;
    if (j == 0) jobs->first[0] = 0;
    jobs->first[j + 1] = jobs->first[j] + (int)fb;
    jobs->F[j] = (const short*)F; jobs->planes[j] = (unsigned char*)planes;
    jobs->layout[j] = {g.C, g.R, g.S, g.K, s.cu, s.cchunks, s.kc_pad, s.ntn, s.bn, s.kt, s.kp,
                            s.gh, s.gw, g.str_h, g.str_w, s.wh, s.ww,
                            g.bprop, s.off_h, s.off_w, g.pad_h, g.pad_w};
    return B2_OK;
}

int run_filter_jobs(const FilterJobs& jobs, cudaStream_t st) {
    B2_CUDA(b2::launch_after(filter_planes_kernel, dim3((unsigned)jobs.first[jobs.n]), 256, 0, st, jobs));
    return B2_OK;
}

int implicit_filter_planes(const void* F, const ConvGeom& g, const ImplicitShape& s, void* planes,
                           cudaStream_t st) {
    FilterJobs jobs = {};
    int rc = add_filter_job(&jobs, F, g, s, planes);
    return rc ? rc : run_filter_jobs(jobs, st);
}

int implicit_tiles(const void* act_planes, const void* filt_planes, void* O, const ConvGeom& g,
                   const ImplicitShape& s, const b2_flex_scale* table, int slotI, int slotF,
                   int slotO, int* stats, unsigned long long* probe_out, int* status, int probe,
                   cudaStream_t st, const b2_conv_epilogue* epi = nullptr) {
    int rc = get_encode();
    if (rc) return rc;
    B2_REQUIRE((((uintptr_t)act_planes | (uintptr_t)filt_planes) & 1023) == 0,
               "operand planes must be 1024-byte aligned");
    void* A0 = (void*)act_planes; void* A1 = (unsigned char*)act_planes + s.act_plane;
    CUtensorMap mI0, mI1, mB;
    if ((rc = make_map_4d(&mI0, A0, g, s.cu, s.wh, s.ww))) return rc;
    if ((rc = make_map_4d(&mI1, A1, g, s.cu, s.wh, s.ww))) return rc;
    if ((rc = make_map(&mB, (void*)filt_planes, s.ntn * 2 * s.bn, s.kp, 1, 2 * s.bn))) return rc;
    ConvTileParams p;
    p.P = g.P; p.Q = g.Q; p.N = g.N; p.K = g.K;
    p.off_h = s.off_h; p.off_w = s.off_w; p.step_h = s.step_h; p.step_w = s.step_w;
    p.cu = s.cu; p.cchunks = s.cchunks; p.kc_pad = s.kc_pad;
    p.box_bytes = s.cu * s.wh * s.ww * 128;
    p.gh = s.gh; p.gw = s.gw; p.tq = (g.Q + s.gw - 1) / s.gw;
    p.gw_log = s.gw == 4 ? 2 : s.gw == 2 ? 1 : 0;
    p.npanels = s.npanels; p.nstages = s.nstages;
    p.bn = s.bn; p.kt = s.kt; p.nbuf = s.nbuf; p.tmem_cols = s.tmem_cols;
    p.nblk = image_blocks(g.N);
    p.num_tiles = s.tiles;
    p.ldc = (long long)g.P * g.Q * g.N;
    p.NP = plane_pitch(g.N); p.ldc_planes = (long long)g.P * g.Q * p.NP;
    p.O = O; p.table = table; p.slotA = slotI; p.slotB = slotF; p.slotC = slotO;
    p.stats = stats; p.probe_out = probe_out; p.status = status; p.probe = probe;
    p.vec = ((uintptr_t)O & 15) == 0 && g.N % 8 == 0; p.mask = nullptr;
    p.bias = nullptr; p.residual = nullptr; p.slot_bias = p.slot_res = 0; p.relu = 0;
    p.write_i16 = 1; p.out_planes = nullptr; p.out_plane_bytes = 0;
    if (epi) {
        B2_REQUIRE(!epi->bias || epi->slot_bias >= 0, "bias needs its scale slot");
        B2_REQUIRE(!epi->residual || epi->slot_residual >= 0, "residual needs its scale slot");
        B2_REQUIRE(epi->write_int16 || epi->out_planes, "the fused epilogue stores nothing");
        B2_REQUIRE(!epi->out_planes || ((uintptr_t)epi->out_planes & 15) == 0, "planes alignment");
        p.bias = epi->bias; p.slot_bias = epi->slot_bias;
        p.residual = epi->residual; p.slot_res = epi->slot_residual;
        p.mask = epi->mask;
        p.relu = epi->relu ? 1 : 0;
        p.write_i16 = epi->write_int16 ? 1 : 0;
        p.out_planes = (unsigned char*)epi->out_planes;
        p.out_plane_bytes = (long long)epi->plane_bytes;
        B2_REQUIRE(!epi->out_planes || (epi->plane_bytes & 7) == 0, "planes alignment");
        p.vec = (((uintptr_t)epi->residual | (uintptr_t)epi->mask | (epi->write_int16 ? (uintptr_t)O : 0)) & 15) == 0 &&
                g.N % 8 == 0;
    }
    dim3 grid(p.num_tiles < 148 ? p.num_tiles : 148, s.ntn);
    // a CTA with one or two tiles has no use for more accumulator sets than tiles: with fewer
    // sets, more epilogue warps share the columns of each
    const int per_cta = (p.num_tiles + (int)grid.x - 1) / (int)grid.x;
    if (per_cta < p.nbuf) p.nbuf = per_cta >= 4 ? 4 : per_cta == 3 ? 3 : per_cta == 2 ? 2 : 1;
    p.n_mma = p.nbuf >= 3 ? 3 : p.nbuf;
    if (const char* e = getenv("B2_CONV_ISSUERS")) {      // measurement aid: 1..3
        const int want = atoi(e);
        if (want >= 1 && want < p.n_mma) p.n_mma = want;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(kConvThreads); cfg.dynamicSmemBytes = s.smem; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = getenv("B2_CONV_NO_PDL") ? 0 : 1;
    typedef void (*Kernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const ConvTileParams);
    typedef unsigned long long U64;
#define B2_TAILS(OFF, SHORT, EVEN)                                                               \
    conv_implicit_kernel<OFF, EPI_FUSED, SHORT, EVEN, false>,                                    \
        conv_implicit_kernel<OFF, EPI_RESIDUAL, SHORT, EVEN, false>,                             \
        conv_implicit_kernel<OFF, EPI_FUSED, SHORT, EVEN, true>,                                 \
        conv_implicit_kernel<OFF, EPI_RESIDUAL, SHORT, EVEN, true>
    static const Kernel kernels[] = {
        conv_implicit_kernel<unsigned, EPI_INT, false, false, false>,
        conv_implicit_kernel<unsigned, EPI_INT, true, false, false>,
        conv_implicit_kernel<unsigned, EPI_INT, true, true, false>,
        conv_implicit_kernel<U64, EPI_INT, false, false, false>,
        B2_TAILS(unsigned, false, false), B2_TAILS(unsigned, false, true), B2_TAILS(unsigned, true, true),
        B2_TAILS(U64, false, false)};
#undef B2_TAILS
    // per product |HH| <= 2^14 and |X| <= 2^14 + 2^15
    const bool short_sum = (long long)g.C * g.R * g.S * ((1 << 22) + (1 << 16)) < (1LL << 31);
    const bool wide = (long long)g.K * p.ldc_planes >= (1LL << 32);
    const bool even = !wide && !probe && p.vec && g.N % 128 == 0 && g.K % 8 == 0 && s.kt % 8 == 0 &&
                      g.K % s.kt == 0;
    const int tail = (p.mask ? 2 : 0) + (p.residual ? 1 : 0);
    const int which = !epi ? (wide ? 3 : !short_sum ? 0 : even ? 2 : 1)
                           : wide ? 16 + tail : !even ? 4 + tail : short_sum ? 12 + tail : 8 + tail;
    static bool attr_set = false;
    if (!attr_set) {
        for (size_t i = 0; i < sizeof(kernels) / sizeof(kernels[0]); ++i)
            B2_CUDA(cudaFuncSetAttribute(kernels[i], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kConvSmemMax));
        attr_set = true;
    }
    B2_CUDA(cudaLaunchKernelEx(&cfg, kernels[which], mI0, mI1, mB, p));
    return B2_OK;
}

template <typename T, int MODE>
int run_fprop_implicit(const T* I, const T* F, void* O, const ConvGeom& g,
                       const b2_flex_scale* table, int slotI, int slotF, int slotO, int* stats,
                       void* scratch, size_t scratch_bytes, unsigned long long* probe_out,
                       int* status, int probe, cudaStream_t st) {
    const ImplicitShape s = implicit_shape(g);
    B2_REQUIRE(scratch && scratch_bytes >= s.bytes && ((uintptr_t)scratch & 1023) == 0,
               "convolution needs %zu bytes of 1024-byte aligned scratch, got %zu", s.bytes,
               scratch_bytes);
    unsigned char* base = (unsigned char*)scratch;
    int rc = implicit_split_activations<T, MODE>(I, g, s, base, st);
    if (rc) return rc;
    if ((rc = implicit_filter_planes(F, g, s, base + 2 * s.act_plane, st))) return rc;
    return implicit_tiles(base, base + 2 * s.act_plane, O, g, s, table, slotI, slotF, slotO, stats,
                          probe_out, status, probe, st);
}

template <typename T, int MODE>
int run_fprop(const T* I, const T* F, void* O, const b2_conv_dims* d, const b2_flex_scale* table,
              int slotI, int slotF, int slotO, int* stats, void* scratch, size_t scratch_bytes,
              unsigned long long* probe_out, int* status, int probe, cudaStream_t st) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(I && F && O, "null tensor");
    if (implicit_ok(MODE, g))
        return run_fprop_implicit<T, MODE>(I, F, O, g, table, slotI, slotF, slotO, stats, scratch,
                                           scratch_bytes, probe_out, status, probe, st);
    b2_direct_args direct;
    if (conv_goes_direct(MODE, g, 0, &direct))
        return launch_direct(direct, I, F, O, table, slotI, slotF, slotO, stats, probe_out, status, probe, st);
    const long long rows_ll = (long long)g.M * g.P * g.Q * g.N;
    B2_REQUIRE(rows_ll < (1LL << 31) - 256, "too many output positions");
    B2_REQUIRE((long long)g.C * g.T * g.R * g.S < (1LL << 24), "filter window too large");
    const int rows = (int)rows_ll, kg = g.C * g.T * g.R * g.S;
    if (MODE == MODE_FLEX16) B2_REQUIRE(kg <= 32768, "flex16 convolution needs C*T*R*S <= 32768");
    const Shapes s = shapes_for(MODE, rows, g.K, kg);
    B2_REQUIRE(scratch && scratch_bytes >= s.bytes && ((uintptr_t)scratch & 1023) == 0,
               "convolution needs %zu bytes of 1024-byte aligned scratch, got %zu", s.bytes,
               scratch_bytes);
    unsigned char* base = (unsigned char*)scratch;
    const size_t a_plane = (size_t)s.Mp * s.Kp * s.esize, b_plane = (size_t)s.Np * s.Kp * s.esize;
    {
        B2_REQUIRE((long long)g.C * g.D * g.H * g.W * g.N < (1LL << 31), "input tensor too large");
        im2col_planes_kernel<T, MODE, false><<<s.Mp / 32, 256, 0, st>>>(I, g, rows, kg, s.Mp, s.Kp,
                                                                base, base + a_plane);
        // filters: element (n = k_out, k = kidx) = F[kidx * K + k_out]
        B2_CUDA(cudaGetLastError());
        rc = split_operand<T, MODE>(F, 1, g.K, g.K, kg, s.Np, s.Kp, base + 2 * a_plane,
                                    base + 2 * a_plane + b_plane, 0, nullptr, st);
        if (rc) return rc;
    }
    GemmParams p;
    p.M = rows; p.N = g.K; p.num_kb = 0;
    p.ldc = rows; p.C = O; p.table = table; p.slotA = slotI; p.slotB = slotF; p.slotC = slotO;
    p.stats = stats; p.probe_out = probe_out; p.status = status; p.probe = probe;
    p.c_colmajor = 1;
    p.rowsum = nullptr;
    return launch_on_planes<MODE>(base, s, p, st);
}

// ---- training contractions -------------------------------------------------------------------
// filter planes for bprop: row = c, column = (k*R + r_)*S + s_, value F[((c*R + r_)*S + s_)*K + k]
template <typename T, int MODE>
__global__ void __launch_bounds__(256)
filter_bprop_planes_kernel(const T* __restrict__ F, int C, int RS, int K, int rows_p, int kp,
                           void* __restrict__ plane0, void* __restrict__ plane1) {
    const long long total = (long long)rows_p * kp;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total;
         i += (long long)gridDim.x * 256) {
        const int c = (int)(i / kp), kidx = (int)(i % kp);
        T v = 0;
        if (c < C && kidx < K * RS) {
            const int k = kidx / RS, rs = kidx - k * RS;
            v = F[((long long)c * RS + rs) * K + k];
        }
        if (MODE == MODE_FLEX16) {
            const int m = (int)v, lo = m & 0xff;
            ((signed char*)plane0)[i] = (signed char)((m - lo) >> 8);
            ((unsigned char*)plane1)[i] = (unsigned char)lo;
        } else {
            float hi, lo;
            tf32_split((float)v, hi, lo);
            ((float*)plane0)[i] = hi;
            ((float*)plane1)[i] = lo;
        }
    }
}

// A planes of the update contraction: row = (c*R + r_)*S + s_, column = (p*Q + q)*N + n, value
// I[c, p*str - pad + r_*dil, q*str - pad + s_*dil, n] (zero outside the image).  One thread writes
// 16 (flex16) or 4 (fp32) consecutive columns; they share (p, q) when N is a multiple of that.
template <typename T, int MODE>
__global__ void __launch_bounds__(256)
update_planes_kernel(const T* __restrict__ I, ConvGeom g, int rows, int kg, int rows_p, int kp,
                     void* __restrict__ plane0, void* __restrict__ plane1) {
    constexpr int kPer = MODE == MODE_FLEX16 ? 16 : 4;
    const int upr = kp / kPer;
    const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
    if (idx >= (long long)rows_p * upr) return;
    const int m = (int)(idx / upr), j0 = (int)(idx % upr) * kPer;
    __align__(16) T v[kPer];
#pragma unroll
    for (int e = 0; e < kPer; ++e) v[e] = 0;
    if (m < rows && j0 < kg) {
        const int RS = g.R * g.S, TRS = g.T * RS;
        const int c = m / TRS, trs = m - c * TRS, ft = trs / RS, rs = trs - ft * RS;
        const int fr = rs / g.S, fs = rs - fr * g.S;
        const T* plane = I + (long long)c * g.D * g.H * g.W * g.N;
        const bool fast = (g.N % kPer == 0) && ((uintptr_t)I & 15) == 0;
        if (fast) {
            const int n0 = j0 % g.N, pq = j0 / g.N, q = pq % g.Q, mp = pq / g.Q, pp = mp % g.P;
            const int dd = (mp / g.P) * g.str_d - g.pad_d + ft * g.dil_d;
            const int h = pp * g.str_h - g.pad_h + fr * g.dil_h;
            const int w = q * g.str_w - g.pad_w + fs * g.dil_w;
            if (h >= 0 && h < g.H && w >= 0 && w < g.W && dd >= 0 && dd < g.D) {
                const T* sp = plane + (((long long)dd * g.H + h) * g.W + w) * g.N + n0;
                if (MODE == MODE_FLEX16) {
                    const int4 a = __ldg((const int4*)sp), b = __ldg((const int4*)sp + 1);
                    *(int4*)&v[0] = a;
                    *(int4*)&v[8 % kPer] = b;
                } else {
                    *(float4*)&v[0] = __ldg((const float4*)sp);
                }
            }
        } else {
#pragma unroll
            for (int e = 0; e < kPer; ++e) {
                const int j = j0 + e;
                if (j >= kg) break;
                const int n = j % g.N, pq = j / g.N, q = pq % g.Q, mp = pq / g.Q, pp = mp % g.P;
                const int dd = (mp / g.P) * g.str_d - g.pad_d + ft * g.dil_d;
                const int h = pp * g.str_h - g.pad_h + fr * g.dil_h;
                const int w = q * g.str_w - g.pad_w + fs * g.dil_w;
                if (h >= 0 && h < g.H && w >= 0 && w < g.W && dd >= 0 && dd < g.D)
                    v[e] = plane[(((long long)dd * g.H + h) * g.W + w) * g.N + n];
            }
        }
    }
    const long long o = (long long)m * kp + j0;
    if (MODE == MODE_FLEX16) {
        unsigned hi[4] = {0, 0, 0, 0}, lo[4] = {0, 0, 0, 0};
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
            const int mm = (int)v[e], l = mm & 0xff;
            hi[e >> 2] |= (unsigned)(((mm - l) >> 8) & 0xff) << (8 * (e & 3));
            lo[e >> 2] |= (unsigned)l << (8 * (e & 3));
        }
        *(uint4*)((unsigned char*)plane0 + o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *(uint4*)((unsigned char*)plane1 + o) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    } else {
        float hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) tf32_split((float)v[e % kPer], hi[e], lo[e]);
        *(float4*)((float*)plane0 + o) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        *(float4*)((float*)plane1 + o) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    }
}

inline void fill_params(GemmParams* p, int M, int N, long long ldc, void* C, int colmajor,
                        const b2_flex_scale* table, int slotA, int slotB, int slotC, int* stats,
                        unsigned long long* probe_out, int* status, int probe) {
    p->M = M; p->N = N; p->num_kb = 0; p->ldc = ldc; p->C = C; p->table = table;
    p->slotA = slotA; p->slotB = slotB; p->slotC = slotC; p->stats = stats;
    p->probe_out = probe_out; p->status = status; p->probe = probe; p->c_colmajor = colmajor;
    p->rowsum = nullptr;
}

struct TrainShape { Shapes s; int splits; size_t bytes; };

TrainShape bprop_shape(int mode, const ConvGeom& g) {
    TrainShape t;
    t.s = shapes_for(mode, g.D * g.H * g.W * g.N, g.C, g.K * g.T * g.R * g.S);
    t.splits = pick_splits(mode, t.s, false);
    t.bytes = align1k(t.s.bytes) + splitk_bytes(mode, t.s, t.splits);
    return t;
}

TrainShape update_shape(int mode, const ConvGeom& g) {
    TrainShape t;
    t.s = shapes_for(mode, g.C * g.T * g.R * g.S, g.K, g.M * g.P * g.Q * g.N);
    t.splits = pick_splits(mode, t.s, true);
    t.bytes = align1k(t.s.bytes) + splitk_bytes(mode, t.s, t.splits);
    return t;
}

template <typename T, int MODE>
int run_bprop(const T* E, const T* F, void* GI, const b2_conv_dims* d, const b2_flex_scale* table,
              int slotE, int slotF, int slotG, int* stats, void* scratch, size_t scratch_bytes,
              unsigned long long* probe_out, int* status, int probe, cudaStream_t st) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(E && F && GI, "null tensor");
    ConvGeom gb;
    if (MODE == MODE_FLEX16 && pass_geom(g, 1, &gb)) {
        const ImplicitShape si = implicit_shape(gb);
        B2_REQUIRE(scratch && scratch_bytes >= si.bytes && ((uintptr_t)scratch & 1023) == 0,
                   "convolution bprop needs %zu bytes of 1024-byte aligned scratch, got %zu",
                   si.bytes, scratch_bytes);
        unsigned char* base = (unsigned char*)scratch;
        if ((rc = implicit_split_activations<T, MODE>(E, gb, si, base, st))) return rc;
        if ((rc = implicit_filter_planes(F, gb, si, base + 2 * si.act_plane, st))) return rc;
        return implicit_tiles(base, base + 2 * si.act_plane, GI, gb, si, table, slotE, slotF, slotG,
                              stats, probe_out, status, probe, st);
    }
    b2_direct_args direct;
    if (conv_goes_direct(MODE, g, 1, &direct))
        return launch_direct(direct, E, F, GI, table, slotE, slotF, slotG, stats, probe_out, status, probe, st);
    const long long rows_ll = (long long)g.D * g.H * g.W * g.N;
    B2_REQUIRE(rows_ll < (1LL << 31) - 256 && (long long)g.K * g.M * g.P * g.Q * g.N < (1LL << 31) &&
               (long long)g.K * g.T * g.R * g.S < (1LL << 24), "tensor too large");
    const int rows = (int)rows_ll, kg = g.K * g.T * g.R * g.S;
    const TrainShape t = bprop_shape(MODE, g);
    const Shapes& s = t.s;
    B2_REQUIRE(scratch && scratch_bytes >= t.bytes && ((uintptr_t)scratch & 1023) == 0,
               "convolution bprop needs %zu bytes of 1024-byte aligned scratch, got %zu", t.bytes,
               scratch_bytes);
    unsigned char* base = (unsigned char*)scratch;
    const size_t a_plane = (size_t)s.Mp * s.Kp * s.esize, b_plane = (size_t)s.Np * s.Kp * s.esize;
    im2col_planes_kernel<T, MODE, true><<<s.Mp / 32, 256, 0, st>>>(E, g, rows, kg, s.Mp, s.Kp, base,
                                                                   base + a_plane);
    long long blocks = ((long long)s.Np * s.Kp + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    filter_bprop_planes_kernel<T, MODE><<<(unsigned)blocks, 256, 0, st>>>(
        F, g.C, g.T * g.R * g.S, g.K, s.Np, s.Kp, base + 2 * a_plane, base + 2 * a_plane + b_plane);
    B2_CUDA(cudaGetLastError());
    GemmParams p;
    fill_params(&p, rows, g.C, rows, GI, 1, table, slotE, slotF, slotG, stats, probe_out, status,
                probe);
    return launch_on_planes<MODE>(base, s, p, st, t.splits, base + align1k(s.bytes));
}

// Division of numbers below 2^16 by a divisor up to 2^15: exact with a 32-bit reciprocal rounded up.
struct FastDiv { unsigned d, m; };
inline FastDiv fast_div(int d) { return {(unsigned)d, (unsigned)((0xffffffffULL + d) / d)}; }
__device__ __forceinline__ int fast_quotient(const FastDiv& f, int x) {
    return f.d == 1 ? x : (int)__umulhi((unsigned)x, f.m);
}

// ---- filter gradient on the tile kernel's operands ------------------------------------------------
// U[(c,r,s), k] = sum over (p,q,n) of I[c, p*str-pad+r, q*str-pad+s, n] * E[k, p, q, n].
// One k-block = a tile of gh x gw output pixels x 128 images.  Its A operand is the very box the forward
// kernel loads (rows (c,h,w): the window under the tile for one channel chunk, images along the row:
// K-major here), its B operand the rows (k, pixel) of the error tensor's planes; the product of window
// row (h,w) with pixel (i,j) belongs to the tap (h - i*str, w - j*str), and the epilogue adds these up.
// A CTA owns a channel chunk, a tile of filters and a range of k-blocks (a slice); both operands come as
// (signed high, unsigned low) byte planes, four exact products HH | X | LL.  The CTAs of the other
// slices add their 64-bit sums to the same accumulators with atomics -- whole numbers, so the order does
// not matter -- and the last to arrive rescales, stores, and leaves the accumulators zero for the next
// call: one launch, no partial sums in memory.  Four idle warps sum the error planes for the bias
// gradient while the tensor core works on them (the chunks of one filter tile take the k-blocks in
// turn).
//
// What bounds it: the bytes from L2 to the SMs and the tensor core about equally.  A window is read
// once per tile instead of once per pixel: for 3x3 filters a tile of 2x2 pixels brings 16 rows a channel
// instead of 36 and fills the 128 rows of the operand (8 channels x 16) where single pixels left 56 empty.
// Filter and bias gradient of a 16-channel 3x3 layer at batch 1024 24 us (46 with single pixels; 69
// and a pass for the bias when the operands were split and the slices summed in launches of their own).
// Clusters of slices that sum through distributed shared memory lost more than they saved: of four
// CTAs with this much shared memory only 33 fit.
struct UpdTileParams {
    int tw, nblk, nkb;             // k-block kb = (tile_p*tw + tile_q)*nblk + nb
    int off_h, off_w, step_h, step_w, str_h, str_w;
    int gh, gw, wh, ww, R, S, cu, C, K, cchunks;
    int ntn, kt, bn;               // filter tiles: kt filters x gh*gw pixels in bn rows
    int per, nsplit;               // k-blocks per slice, slices (grid.x)
    FastDiv by_kt, by_rs, by_s;
    int ksteps, nstages, tmem_cols;
    unsigned box_a, box_b;         // bytes of one activation box, of one error box
    unsigned long long* acc;       // [C*R*S][K], then [K] for the bias: zero between calls
    unsigned* arrived;             // [cchunks*ntn], then [ntn]: likewise
    short *U, *bias;               // bias gradient: NULL where it is not wanted
    const b2_flex_scale* table;
    int slotI, slotE, slotU, slotB;
    int* stats;
    unsigned long long* probe_out; // probe: max |sum| of U, of the bias
    int* status;
    int probe;
};

constexpr int kUpdThreads = 512;
constexpr int kUpdMaxStages = 6;
constexpr int kUpdMaxN = 160;                      // columns of one accumulator: three in 512
constexpr int kUpdAPlane = 128 * kKBytes;          // 128 rows of 128 bytes
constexpr int kUpdSmemFixed = 1024 + 256 + kUpdMaxN * 8;

// largest of a block's non-negative values, in thread 0's atomic
template <typename V, typename F>
__device__ __forceinline__ void update_max(V v, F put) {
    for (int o = 16; o > 0; o >>= 1) {
        const V t = __shfl_xor_sync(0xffffffffu, v, o);
        v = t > v ? t : v;
    }
    if ((threadIdx.x & 31) == 0 && v) put(v);
}

__global__ void __launch_bounds__(kUpdThreads, 1)
conv_update_kernel(const __grid_constant__ CUtensorMap mapI0, const __grid_constant__ CUtensorMap mapI1,
                   const __grid_constant__ CUtensorMap mapE0, const __grid_constant__ CUtensorMap mapE1,
                   const UpdTileParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int bn = p.bn, kt = p.kt;
    const int b_plane = bn * kKBytes, stage = 2 * kUpdAPlane + 2 * b_plane;
    unsigned long long* full_bar = (unsigned long long*)(ring + (size_t)p.nstages * stage);
    unsigned long long* empty_bar = full_bar + kUpdMaxStages;
    unsigned long long* tmem_full = empty_bar + kUpdMaxStages;
    unsigned* tmem_holder = (unsigned*)(tmem_full + 1);
    int* fail_flag = (int*)(tmem_holder + 1);
    unsigned* last = (unsigned*)(fail_flag + 1);                 // [2]
    long long* bias_sum = (long long*)((unsigned char*)full_bar + 256);           // [kt]

    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int chunk = blockIdx.y / p.ntn, ktile = blockIdx.y - chunk * p.ntn;
    const int kb0 = blockIdx.x * p.per;
    int mine = p.nkb - kb0;
    if (mine > p.per) mine = p.per;
    const int npix = p.gh * p.gw;

    if (threadIdx.x == 0) {
        prefetch_map(&mapI0); prefetch_map(&mapI1); prefetch_map(&mapE0); prefetch_map(&mapE1);
        for (int s = 0; s < kUpdMaxStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], p.bias ? 6 : 2);
        }
        mbar_init(tmem_full, 2);
        *fail_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < kt; i += kUpdThreads) bias_sum[i] = 0;
    if (warp == 1) {
        tmem_alloc(tmem_holder, p.tmem_cols);
        // (not before this CTA holds its tensor memory, or it and the next kernel's could each wait for
        // what the other has)
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = (unsigned)warp_uniform((int)*tmem_holder);

    if (warp == 0) {
        if (elect_one()) {
            int s = 0;
            unsigned empty_parity = 1;
            int nb = kb0 % p.nblk, pq = kb0 / p.nblk, q = pq % p.tw, pp = pq / p.tw;
            for (int i = 0; i < mine; ++i) {
                if (!mbar_wait_relaxed(&empty_bar[s], empty_parity)) { atomicExch(fail_flag, 1); break; }
                unsigned char* sa = ring + (size_t)s * stage;
                mbar_expect_tx(&full_bar[s], 2 * p.box_a + 2 * p.box_b);
                const int w0 = q * p.step_w + p.off_w, h0 = pp * p.step_h + p.off_h;
                tma_load_4d(sa, &mapI0, nb * 128, w0, h0, chunk * p.cu, &full_bar[s]);
                tma_load_4d(sa + kUpdAPlane, &mapI1, nb * 128, w0, h0, chunk * p.cu, &full_bar[s]);
                unsigned char* sb = sa + 2 * kUpdAPlane;
                tma_load_4d(sb, &mapE0, nb * 128, q * p.gw, pp * p.gh, ktile * kt, &full_bar[s]);
                tma_load_4d(sb + b_plane, &mapE1, nb * 128, q * p.gw, pp * p.gh, ktile * kt, &full_bar[s]);
                if (++s == p.nstages) { s = 0; empty_parity ^= 1u; }
                if (++nb == p.nblk) {
                    nb = 0;
                    if (++q == p.tw) { q = 0; ++pp; }
                }
            }
        }
    } else if (warp == 1 || warp == 2) {
        // two issuing threads, for different accumulators: HH and LL, X (one thread alone took 70
        // cycles an instruction)
        const bool cross = warp == 2;
        if (elect_one()) {
            const unsigned id_h = make_idesc_n(2, 1, cross ? 0 : 1, bn), id_l = make_idesc_n(2, 0, cross ? 1 : 0, bn);
            const unsigned acc_h = tmem_base + (cross ? bn : 0), acc_l = tmem_base + (cross ? bn : 2 * bn);
            // matrix descriptors: only the low word (start address in 16-byte units) changes
            const unsigned long long dsc = make_smem_desc(ring) & ~0x3fffULL;
            const unsigned stage_units = (unsigned)(stage >> 4), a_units = kUpdAPlane >> 4,
                           b_units = (unsigned)(b_plane >> 4), ring_at = (smem_u32(ring) >> 4) & 0x3FFF;
            const unsigned bh = 2 * a_units + (cross ? b_units : 0), bl = 2 * a_units + (cross ? 0 : b_units);
            const int ksteps = p.ksteps;
            unsigned accumulate = 0, parity = 0, at = ring_at;
            int s = 0;
            for (int i = 0; i < mine; ++i) {
                if (!mbar_wait(&full_bar[s], parity)) { atomicExch(fail_flag, 1); break; }
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (k >= ksteps) break;
                    tc_mma<MODE_FLEX16>(acc_h, dsc | (at + 2 * k), dsc | (at + bh + 2 * k), id_h, accumulate);
                    tc_mma<MODE_FLEX16>(acc_l, dsc | (at + a_units + 2 * k), dsc | (at + bl + 2 * k), id_l,
                                        cross ? 1u : accumulate);
                    accumulate = 1;
                }
                tc_commit(&empty_bar[s]);
                at += stage_units;
                if (++s == p.nstages) { s = 0; parity ^= 1u; at = ring_at; }
            }
            tc_commit(tmem_full);
        }
    } else if (warp >= 4 && warp < 8 && p.bias) {
        // sums of the error rows: thread t takes the 16-byte units t, t + 128, ..., whose rows
        // are t/8 + 16*m
        const int t = threadIdx.x - 128;
        constexpr int kMost = kUpdMaxN / 16;
        int hi[kMost], lo[kMost];
#pragma unroll
        for (int m = 0; m < kMost; ++m) hi[m] = lo[m] = 0;
        int s = 0, turn = 0;
        unsigned parity = 0;
        bool ok = true;
        for (int i = 0; i < mine; ++i) {
            if (ok && !mbar_wait_relaxed(&full_bar[s], parity)) { atomicExch(fail_flag, 1); ok = false; }
            if (turn == chunk && ok) {
                const unsigned char* sb = ring + (size_t)s * stage + 2 * kUpdAPlane + t * 16;
#pragma unroll
                for (int m = 0; m < kMost; ++m) {
                    if (m * 16 >= bn) break;
                    const int4 h = *(const int4*)(sb + m * 2048);
                    const uint4 l = *(const uint4*)(sb + b_plane + m * 2048);
                    hi[m] = __dp4a(h.x, 0x01010101, hi[m]); lo[m] = (int)__dp4a(l.x, 0x01010101u, (unsigned)lo[m]);
                    hi[m] = __dp4a(h.y, 0x01010101, hi[m]); lo[m] = (int)__dp4a(l.y, 0x01010101u, (unsigned)lo[m]);
                    hi[m] = __dp4a(h.z, 0x01010101, hi[m]); lo[m] = (int)__dp4a(l.z, 0x01010101u, (unsigned)lo[m]);
                    hi[m] = __dp4a(h.w, 0x01010101, hi[m]); lo[m] = (int)__dp4a(l.w, 0x01010101u, (unsigned)lo[m]);
                }
            }
            if (++turn == p.cchunks) turn = 0;
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty_bar[s]);
            if (++s == p.nstages) { s = 0; parity ^= 1u; }
        }
#pragma unroll
        for (int m = 0; m < kMost; ++m) {
            if (m * 16 >= bn) break;
            long long v = 256LL * hi[m] + lo[m];
            for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const int row = (t >> 3) + 16 * m;
            if ((t & 7) == 0 && row < kt * npix && ok)
                atomicAdd((unsigned long long*)bias_sum + row / npix, (unsigned long long)v);
        }
    }
    __syncwarp();
    __syncthreads();                                  // (every reader is done with the ring)

    // exact sums of this slice: tensor memory -> shared memory [row][column]
    bool ok = mbar_wait_relaxed(tmem_full, 0);
    if (!ok) atomicExch(fail_flag, 1);
    tc_fence_after();
    long long* red = (long long*)ring;
    const int pitch = bn + 1;                         // odd: the 32 rows of a store fall into different banks
    {
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const unsigned a0 = tmem_base + ((unsigned)(quarter * 32) << 16);
        for (int c0 = (warp >> 2) * 8; c0 < bn; c0 += 32) {
            unsigned hh[8], xx[8], ll[8];
            tmem_ld8(a0 + c0, hh); tmem_ld8(a0 + bn + c0, xx); tmem_ld8(a0 + 2 * bn + c0, ll);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 8; ++j)
                red[row * pitch + c0 + j] = mine <= 0 ? 0 :
                    ((long long)(int)hh[j] << 16) + ((long long)(int)xx[j] << 8) + (long long)ll[j];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, p.tmem_cols);
    }
    ok = *fail_flag == 0;
    const int rs = p.R * p.S, n_out = p.cu * rs * kt;
    unsigned long long* bias_acc = p.acc + (long long)p.C * rs * p.K + ktile * kt;
    // ... added up per tap in shared memory, then onto the accumulators: rows of 16-byte multiples by bulk
    // reductions (a 64-bit atomic takes its SM four cycles a value: 7500 cycles for a 64-channel tile,
    // 1200 this way)
    long long* sum = red + 128 * pitch;                          // (16-byte aligned: 128 is even)
    const int rows = (p.C - chunk * p.cu < p.cu ? p.C - chunk * p.cu : p.cu) * rs;
    const int width = p.K - ktile * kt < kt ? p.K - ktile * kt : kt;
    const bool bulk = ((p.K | kt) & 1) == 0;
    unsigned long long* acc = p.acc + (long long)chunk * p.cu * rs * p.K + ktile * kt;
    for (int i = threadIdx.x; i < rows * kt && ok; i += kUpdThreads) {
        const int t = fast_quotient(p.by_kt, i), k = i - t * kt, c = fast_quotient(p.by_rs, t), tap = t - c * rs;
        const int r = fast_quotient(p.by_s, tap), s = tap - r * p.S;
        const long long* at = red + ((c * p.wh + r) * p.ww + s) * pitch + k * npix;
        long long v = 0;
        for (int a = 0; a < p.gh; ++a)
            for (int b = 0; b < p.gw; ++b) v += at[(a * p.str_h * p.ww + b * p.str_w) * pitch + a * p.gw + b];
        if (bulk) sum[i] = v;
        else if (k < width && v) atomicAdd(acc + (long long)t * p.K + k, (unsigned long long)v);
    }
    if (bulk) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        const bool whole = kt == p.K;                     // then the tile is one piece
        if (ok)
            for (int t = threadIdx.x; t < (whole ? 1 : rows); t += kUpdThreads)
                asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.u64 [%0], [%1], %2;"
                             ::"l"(acc + (long long)t * p.K), "r"(smem_u32(sum + t * kt)),
                               "r"((whole ? rows * kt : width) * 8) : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.global;" ::: "memory");
    }
    if (p.bias)
        for (int k = threadIdx.x; k < kt && ktile * kt + k < p.K; k += kUpdThreads)
            if (bias_sum[k] && ok) atomicAdd(bias_acc + k, (unsigned long long)bias_sum[k]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned* tile = p.arrived + blockIdx.y;
        unsigned* col = p.arrived + p.cchunks * p.ntn + ktile;
        last[0] = atomicAdd(tile, 1u) == (unsigned)p.nsplit - 1u;
        if (last[0]) *tile = 0;
        last[1] = p.bias && atomicAdd(col, 1u) == (unsigned)(p.nsplit * p.cchunks) - 1u;
        if (last[1]) *col = 0;
        if (*fail_flag && p.status) atomicExch(p.status, 1);
    }
    __syncthreads();
    if (!last[0] && !last[1]) return;
    __threadfence();
    const float scale_e = p.table[p.slotE].scale;
    if (last[0]) {
        const int sh = -ilogbf(p.table[p.slotI].scale * scale_e * (p.probe ? 1.0f : p.table[p.slotU].inv_scale));
        int stat = 0;
        unsigned long long pmax = 0;
        constexpr int kBatch = 8;                         // loads in flight
        for (int i0 = threadIdx.x; i0 < n_out; i0 += kBatch * kUpdThreads) {
            long long at[kBatch], v[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                const int i = i0 + j * kUpdThreads, t = fast_quotient(p.by_kt, i), kg = ktile * kt + i - t * kt;
                const long long row = (long long)chunk * p.cu * rs + t;
                at[j] = i < n_out && row < (long long)p.C * rs && kg < p.K ? row * p.K + kg : -1;
                v[j] = at[j] >= 0 ? (long long)__ldcg(p.acc + at[j]) : 0;
            }
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                if (at[j] < 0) continue;
                p.acc[at[j]] = 0;
                if (p.probe) {
                    const unsigned long long m = (unsigned long long)(v[j] < 0 ? -v[j] : v[j]);
                    pmax = m > pmax ? m : pmax;
                } else {
                    const int q = rescale_i64(v[j], sh), m = q < 0 ? -q : q;
                    stat = m > stat ? m : stat;
                    p.U[at[j]] = (short)q;
                }
            }
        }
        if (p.probe) update_max(pmax, [&](unsigned long long m) { atomicMax(p.probe_out, m); });
        else update_max(stat, [&](int m) { atomicMax(p.stats + p.slotU, m); });
    }
    if (last[1]) {
        // an elementwise sum's quantisation: truncation toward zero
        const int sh = -ilogbf(scale_e * (p.probe ? 1.0f : p.table[p.slotB].inv_scale));
        int stat = 0;
        unsigned long long pmax = 0;
        for (int k = threadIdx.x; k < kt && ktile * kt + k < p.K; k += kUpdThreads) {
            const long long v = (long long)__ldcg(bias_acc + k);
            bias_acc[k] = 0;
            const unsigned long long m = (unsigned long long)(v < 0 ? -v : v);
            if (p.probe) {
                pmax = m > pmax ? m : pmax;
                continue;
            }
            unsigned long long q = sh >= 63 ? 0 : sh >= 0 ? m >> sh : m >= 32768 || sh <= -16 ? (m ? 32768 : 0) : m << -sh;
            const unsigned long long most = v < 0 ? 32768 : 32767;
            q = q > most ? most : q;
            stat = (int)q > stat ? (int)q : stat;
            p.bias[ktile * kt + k] = (short)(v < 0 ? -(int)q : (int)q);
        }
        if (p.probe) update_max(pmax, [&](unsigned long long m) { atomicMax(p.probe_out + 1, m); });
        else update_max(stat, [&](int m) { atomicMax(p.stats + p.slotB, m); });
    }
}

struct UpdShape {
    bool ok;
    int gh, gw, wh, ww, cu, cchunks, ntn, kt, bn, tmem_cols, ksteps, nstages, smem, tw, nblk, nkb, per, nsplit;
    size_t act_plane, err_plane, acc_bytes;
    long long cost;
};

// Cost in cycles, fitted to measured launches: a k-block takes what the tensor core needs for its
// products, or its bytes from L2 at 56 a cycle; set-up, the sums' way to memory and the last CTA's work
// take 8 us, and more with the columns and outputs of a tile.
UpdShape update_shape_for(const ConvGeom& g, int gh, int gw) {
    UpdShape u = {};
    u.gh = gh; u.gw = gw; u.wh = (gh - 1) * g.str_h + g.R; u.ww = (gw - 1) * g.str_w + g.S;
    const int win = u.wh * u.ww, npix = gh * gw;
    const long long th = (g.P + gh - 1) / gh, nblk = image_blocks(g.N);
    u.tw = (g.Q + gw - 1) / gw; u.nblk = (int)nblk;
    if (win > 128 || th * u.tw * nblk >= (1LL << 30)) return u;
    const int cu_max = 128 / win;
    u.cchunks = (g.C + cu_max - 1) / cu_max;
    u.cu = (g.C + u.cchunks - 1) / u.cchunks;
    const int kt_max = npix == 1 ? 96 : kUpdMaxN / npix;
    u.ntn = (g.K + kt_max - 1) / kt_max;
    u.kt = (g.K + u.ntn - 1) / u.ntn;
    u.bn = round_up(u.kt * npix, 16);
    u.tmem_cols = 32;
    while (u.tmem_cols < 3 * u.bn) u.tmem_cols *= 2;
    const int stage = 2 * kUpdAPlane + 2 * u.bn * kKBytes;
    u.nstages = (kConvSmemMax - kUpdSmemFixed) / stage;
    if (u.nstages > kUpdMaxStages) u.nstages = kUpdMaxStages;
    if (u.nstages < 2 || (long long)u.cchunks * u.ntn > 65535) return u;
    u.smem = kUpdSmemFixed + u.nstages * stage;
    // (the ring holds the sums afterwards, by row and column and by output)
    if (128 * (u.bn + 1) * 8 + u.cu * g.R * g.S * u.kt * 8 > u.nstages * stage) return u;
    u.nkb = (int)(th * u.tw * nblk);
    const int images = g.N < 128 ? g.N : 128;
    u.ksteps = (images + 31) / 32;
    const int cols = u.cchunks * u.ntn;
    int slices = cols < 148 ? 148 / cols : 1;
    if (slices < (u.nkb + 255) / 256) slices = (u.nkb + 255) / 256;   // int32 sums: exact up to 32768 terms
    u.per = (u.nkb + slices - 1) / slices;
    u.nsplit = (u.nkb + u.per - 1) / u.per;
    const long long mma = 16LL * u.ksteps / 4 * (u.bn / 2 > 32 + u.bn / 4 ? u.bn / 2 : 32 + u.bn / 4);
    const long long bytes = 2LL * images * (u.cu * win + u.kt * npix) / 56;
    u.cost = ((long long)cols * u.nsplit + 147) / 148 *
             (u.per * ((mma > bytes ? mma : bytes) + 60) + 15500 + 48 * u.bn + 2LL * u.cu * g.R * g.S * u.kt);
    u.act_plane = plane_size(g.C, g.H, g.W, g.N);
    u.err_plane = plane_size(g.K, g.P, g.Q, g.N);
    u.acc_bytes = align1k((((size_t)g.C * g.R * g.S + 1) * g.K) * 8 + (size_t)(cols + u.ntn) * 4);
    u.ok = true;
    return u;
}

UpdShape update_implicit_shape(int mode, const ConvGeom& g) {
    UpdShape best = {};
    if (mode != MODE_FLEX16 || g.dil_h != 1 || g.dil_w != 1 || !flat_depth(g) || getenv("B2_CONV_IM2COL"))
        return best;
    for (int gh = 1; gh <= 2; ++gh)
        for (int gw = 1; gw <= 2; ++gw) {
            const UpdShape u = update_shape_for(g, gh, gw);
            if (u.ok && (!best.ok || u.cost < best.cost)) best = u;
        }
    return best;
}

struct UpdOut {
    void *U, *bias;
    const b2_flex_scale* table;
    int slotI, slotE, slotU, slotB;
    int* stats;
    unsigned long long* probe_out;
    int* status;
    int probe;
};

int run_update_planes(const void* act_planes, const void* err_planes, void* acc, const ConvGeom& g,
                      const UpdShape& u, const UpdOut& o, cudaStream_t st) {
    int rc = get_encode();
    if (rc) return rc;
    B2_REQUIRE((((uintptr_t)act_planes | (uintptr_t)err_planes | (uintptr_t)acc) & 1023) == 0,
               "planes and workspace must be 1024-byte aligned");
    unsigned char *I0 = (unsigned char*)act_planes, *E0 = (unsigned char*)err_planes;
    ConvGeom e = g;
    e.C = g.K; e.H = g.P; e.W = g.Q;
    CUtensorMap mI0, mI1, mE0, mE1;
    if ((rc = make_map_4d(&mI0, I0, g, u.cu, u.wh, u.ww))) return rc;
    if ((rc = make_map_4d(&mI1, I0 + u.act_plane, g, u.cu, u.wh, u.ww))) return rc;
    if ((rc = make_map_4d(&mE0, E0, e, u.kt, u.gh, u.gw))) return rc;
    if ((rc = make_map_4d(&mE1, E0 + u.err_plane, e, u.kt, u.gh, u.gw))) return rc;
    UpdTileParams p;
    p.tw = u.tw; p.nblk = u.nblk; p.nkb = u.nkb;
    p.off_h = -g.pad_h; p.off_w = -g.pad_w; p.step_h = u.gh * g.str_h; p.step_w = u.gw * g.str_w;
    p.str_h = g.str_h; p.str_w = g.str_w;
    p.gh = u.gh; p.gw = u.gw; p.wh = u.wh; p.ww = u.ww; p.R = g.R; p.S = g.S;
    p.cu = u.cu; p.C = g.C; p.K = g.K; p.cchunks = u.cchunks;
    p.ntn = u.ntn; p.kt = u.kt; p.bn = u.bn; p.per = u.per; p.nsplit = u.nsplit;
    p.by_kt = fast_div(u.kt); p.by_rs = fast_div(g.R * g.S); p.by_s = fast_div(g.S);
    p.ksteps = u.ksteps; p.nstages = u.nstages; p.tmem_cols = u.tmem_cols;
    p.box_a = (unsigned)(u.cu * u.wh * u.ww * kKBytes); p.box_b = (unsigned)(u.kt * u.gh * u.gw * kKBytes);
    p.acc = (unsigned long long*)acc;
    p.arrived = (unsigned*)(p.acc + ((size_t)g.C * g.R * g.S + 1) * g.K);
    p.U = (short*)o.U; p.bias = (short*)o.bias; p.table = o.table;
    p.slotI = o.slotI; p.slotE = o.slotE; p.slotU = o.slotU; p.slotB = o.slotB;
    p.stats = o.stats; p.probe_out = o.probe_out; p.status = o.status; p.probe = o.probe;
    static bool attr_set = false;
    if (!attr_set) {
        B2_CUDA(cudaFuncSetAttribute(conv_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kConvSmemMax));
        attr_set = true;
    }
    B2_CUDA(b2::launch_after(conv_update_kernel, dim3(u.nsplit, u.cchunks * u.ntn), kUpdThreads, u.smem, st, mI0,
                             mI1, mE0, mE1, p));
    return B2_OK;
}

// from int16 tensors: whole tiles of 128 images, as the entry point's scratch has always been sized
inline bool update_goes_in_planes(int mode, const ConvGeom& g, UpdShape* u) {
    *u = update_implicit_shape(mode, g);
    return u->ok && g.N % 128 == 0;
}
inline size_t update_planes_bytes(const UpdShape& u) { return 2 * u.act_plane + 2 * u.err_plane + u.acc_bytes; }

int run_update_implicit(const short* I, const short* E, const ConvGeom& g, const UpdShape& u, const UpdOut& o,
                        void* scratch, size_t scratch_bytes, cudaStream_t st) {
    B2_REQUIRE(scratch && scratch_bytes >= update_planes_bytes(u) && ((uintptr_t)scratch & 1023) == 0,
               "convolution update needs %zu bytes of 1024-byte aligned scratch, got %zu",
               update_planes_bytes(u), scratch_bytes);
    unsigned char* base = (unsigned char*)scratch;
    unsigned char* eplanes = base + 2 * u.act_plane;
    unsigned char* acc = eplanes + 2 * u.err_plane;
    int rc = split_to_planes(I, g.C, g.H, g.W, g.N, base, u.act_plane, st);
    if (rc) return rc;
    if ((rc = split_to_planes(E, g.K, g.P, g.Q, g.N, eplanes, u.err_plane, st))) return rc;
    B2_CUDA(cudaMemsetAsync(acc, 0, u.acc_bytes, st));
    return run_update_planes(base, eplanes, acc, g, u, o, st);
}

// the fp32 kernel that converts on the way in; its scratch, 0 where it does not take the problem
inline size_t update_f32_scratch(int mode, const ConvGeom& g, b2_update_f32* d) {
    if (mode != MODE_F32X3 || g.dil_h != 1 || g.dil_w != 1 || !flat_depth(g) || getenv("B2_CONV_IM2COL")) return 0;
    *d = {g.C, g.H, g.W, g.N, g.K, g.R, g.S, g.P, g.Q, g.pad_h, g.pad_w, g.str_h, g.str_w};
    return b2_update_f32_scratch(*d);
}

template <typename T, int MODE>
int run_update(const T* I, const T* E, void* U, const b2_conv_dims* d, const b2_flex_scale* table,
               int slotI, int slotE, int slotU, int* stats, void* scratch, size_t scratch_bytes,
               unsigned long long* probe_out, int* status, int probe, cudaStream_t st) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(I && E && U, "null tensor");
    {
        UpdShape u;
        if (update_goes_in_planes(MODE, g, &u)) {
            const UpdOut o = {U, nullptr, table, slotI, slotE, slotU, -1, stats, probe_out, status, probe};
            return run_update_implicit((const short*)I, (const short*)E, g, u, o, scratch, scratch_bytes, st);
        }
    }
    b2_update_f32 f32;
    if (const size_t need = update_f32_scratch(MODE, g, &f32)) {
        B2_REQUIRE(scratch && scratch_bytes >= need && ((uintptr_t)scratch & 1023) == 0,
                   "convolution update needs %zu bytes of 1024-byte aligned scratch, got %zu", need, scratch_bytes);
        return b2_update_f32_launch(f32, (const float*)I, (const float*)E, (float*)U, scratch, status, st);
    }
    const long long kg_ll = (long long)g.M * g.P * g.Q * g.N;
    B2_REQUIRE(kg_ll < (1LL << 31) - 256 && (long long)g.C * g.D * g.H * g.W * g.N < (1LL << 31) &&
               (long long)g.C * g.T * g.R * g.S < (1LL << 24), "tensor too large");
    const int rows = g.C * g.T * g.R * g.S, kg = (int)kg_ll;
    const TrainShape t = update_shape(MODE, g);
    const Shapes& s = t.s;
    B2_REQUIRE(scratch && scratch_bytes >= t.bytes && ((uintptr_t)scratch & 1023) == 0,
               "convolution update needs %zu bytes of 1024-byte aligned scratch, got %zu", t.bytes,
               scratch_bytes);
    unsigned char* base = (unsigned char*)scratch;
    const size_t a_plane = (size_t)s.Mp * s.Kp * s.esize, b_plane = (size_t)s.Np * s.Kp * s.esize;
    const long long units = (long long)s.Mp * (s.Kp / (MODE == MODE_FLEX16 ? 16 : 4));
    update_planes_kernel<T, MODE><<<(unsigned)((units + 255) / 256), 256, 0, st>>>(
        I, g, rows, kg, s.Mp, s.Kp, base, base + a_plane);
    B2_CUDA(cudaGetLastError());
    // E is [K][(p,q,n)]: already the K-major B operand
    rc = split_operand<T, MODE>(E, (long long)kg, 1, g.K, kg, s.Np, s.Kp, base + 2 * a_plane,
                                base + 2 * a_plane + b_plane, 0, nullptr, st);
    if (rc) return rc;
    GemmParams p;
    fill_params(&p, rows, g.K, g.K, U, 0, table, slotI, slotE, slotU, stats, probe_out, status,
                probe);
    return launch_on_planes<MODE>(base, s, p, st, t.splits, base + align1k(s.bytes));
}

// ---- average pooling over H, W windows (C and D windows of 1) ------------------------------------
// out[c,p,q,n] = mean over the part of the window inside the image (the numpy reference takes
// np.mean of the clipped slice, ngraph/transformers/cpu/cpuengine.py:296-305).  flex16: the output
// shares the input's exponent (ngraph/transformers/passes/flexpass.py:40-48), so mantissas are
// averaged and rounded to nearest even.
template <typename T, bool MAX>
__global__ void __launch_bounds__(256)
pool_kernel(const T* __restrict__ I, T* __restrict__ O, int C, int H, int W, int N, int P, int Q,
            int R, int S, int pad_h, int pad_w, int str_h, int str_w, int* stats) {
    after_earlier_kernels();
    // a block takes 32 consecutive results (consecutive images: coalesced); its eight warps each
    // add every eighth element of the window, the eight partial sums are combined in warp order
    __shared__ float part[8][32];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const long long total = (long long)C * P * Q * N;
    const long long units = (total + 31) / 32;
    int stat = 0;
    for (long long u = blockIdx.x; u < units; u += gridDim.x) {
        const long long i = u * 32 + tx;
        const bool live = i < total;
        float acc = MAX ? -INFINITY : 0.0f;
        int cnt = 1;
        if (live) {
            const int n = (int)(i % N);
            long long t = i / N;
            const int q = (int)(t % Q); t /= Q;
            const int p = (int)(t % P);
            const int c = (int)(t / P);
            const int h0 = max(p * str_h - pad_h, 0), h1 = min(p * str_h - pad_h + R, H);
            const int w0 = max(q * str_w - pad_w, 0), w1 = min(q * str_w - pad_w + S, W);
            const int wlen = max(w1 - w0, 0), area = max(h1 - h0, 0) * wlen;
            cnt = max(area, 1);
            for (int e = ty; e < area; e += 8) {
                const int h = h0 + e / wlen, w = w0 + e % wlen;
                const float v = (float)I[(((long long)c * H + h) * W + w) * N + n];
                acc = MAX ? fmaxf(acc, v) : acc + v;
            }
        }
        part[ty][tx] = acc;
        __syncthreads();
        if (ty == 0 && live) {
            float sum = part[0][tx];
#pragma unroll
            for (int k = 1; k < 8; ++k) sum = MAX ? fmaxf(sum, part[k][tx]) : sum + part[k][tx];
            // (a window that lies entirely in the padding has no element: 0, as the mean gives)
            const float mean = MAX ? (sum == -INFINITY ? 0.0f : sum) : sum / (float)cnt;
            if (sizeof(T) == 2) {
                const int m = __float2int_rn(mean);
                stat = max(stat, m < 0 ? -m : m);
                O[i] = (T)m;
            } else {
                O[i] = (T)mean;
            }
        }
        __syncthreads();
    }
    if (sizeof(T) == 2 && stats && ty == 0) {
        for (int o = 16; o > 0; o >>= 1) stat = max(stat, __shfl_xor_sync(0xffffffffu, stat, o));
        if (tx == 0 && stat) atomicMax(stats, stat);
    }
}

}  // namespace

extern "C" int b2_conv_fprop_scratch_bytes(int32_t flex, const b2_conv_dims* d, size_t* bytes) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(bytes, "null argument");
    const int mode = flex ? MODE_FLEX16 : MODE_F32X3;
    b2_direct_args direct;
    *bytes = implicit_ok(mode, g) ? implicit_shape(g).bytes
             : conv_goes_direct(mode, g, 0, &direct)
                 ? 0 : shapes_for(mode, g.M * g.P * g.Q * g.N, g.K, g.C * g.T * g.R * g.S).bytes;
    return B2_OK;
}

extern "C" int b2_conv_launches(int32_t flex, const b2_conv_dims* d, int32_t pass, int32_t* launches) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(launches && pass >= 0 && pass <= 2, "bad argument");
    const int mode = flex ? MODE_FLEX16 : MODE_F32X3;
    ConvGeom gp;
    b2_direct_args direct;
    UpdShape u;
    b2_update_f32 f32;
    if (pass == 2)
        *launches = update_f32_scratch(mode, g, &f32) ? b2_update_f32_launches(f32) : !update_goes_in_planes(mode, g, &u) && update_shape(mode, g).splits > 1 ? 4 : 3;
    else
        *launches = !(flex && pass_geom(g, pass, &gp)) && conv_goes_direct(mode, g, pass, &direct) ? 1 : 3;
    return B2_OK;
}

extern "C" int b2_conv_fprop_f32_fused(const float* I, const float* F, float* O, const b2_conv_dims* d,
                                       const float* bias, const float* residual, int32_t relu,
                                       int32_t* status, void* stream) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(I && F && O, "null tensor");
    b2_direct_args direct;
    B2_REQUIRE(conv_goes_direct(MODE_F32X3, g, 0, &direct), "this convolution takes no fused tail");
    direct.bias = bias; direct.residual = residual; direct.relu = relu ? 1 : 0;
    return launch_direct(direct, I, F, O, nullptr, 0, 0, 0, nullptr, nullptr, status, 0, (cudaStream_t)stream);
}

extern "C" int b2_conv_f32_plan(const b2_conv_dims* d, int32_t pass, int32_t tiles, b2_conv_plan_info* plan) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(plan && (pass == 0 || pass == 1), "bad argument");
    *plan = {};
    b2_direct_args a;
    if (!(tiles ? conv_goes_staged(g, pass, &a) : conv_goes_direct(MODE_F32X3, g, pass, &a))) return B2_OK;
    b2_gemm_plan_info p;
    b2_direct_plan(a, &p);
    *plan = {a.g.gh, a.g.gw, p.tile_n, p.slices, (a.K + 31) / 32, b2_direct_in_one_sum(a)};
    return B2_OK;
}

extern "C" int b2_conv_f32_sums(const b2_conv_dims* d, int32_t pass, b2_conv_sums_info* sums) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(sums && (pass == 0 || pass == 1), "bad argument");
    *sums = {};
    b2_direct_args a, other;
    if (!conv_goes_staged(g, pass, &a, &other)) return B2_OK;
    const int large = b2_direct_in_one_sum(a);
    const bool gathers = b2_gather_streams(a);
    *sums = {gathers ? B2_CONV_GATHER : B2_CONV_DIRECT, large, gathers ? b2_gather_plan(a).small : large, 0, b2_direct_loss(a),
             b2_direct_loss(other)};
    return B2_OK;
}

extern "C" int b2_conv_filter_tiles_info(const b2_conv_dims* d, int32_t pass, size_t* bytes) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(bytes && (pass == 0 || pass == 1), "bad argument");
    b2_direct_args direct;
    *bytes = conv_goes_staged(g, pass, &direct) ? b2_direct_staged_bytes(direct) : 0;
    return B2_OK;
}

extern "C" int b2_conv_filter_tiles(const b2_conv_filter_job* jobs, int32_t n, int32_t* launches, void* stream) {
    B2_REQUIRE(jobs && n >= 0 && launches, "bad argument");
    *launches = 0;
    for (int32_t at = 0; at < n; at += kStageJobs) {
        b2_stage_job list[kStageJobs];
        const int m = n - at < kStageJobs ? n - at : kStageJobs;
        for (int j = 0; j < m; ++j) {
            const b2_conv_filter_job& job = jobs[at + j];
            ConvGeom g;
            int rc = geom_from(&job.dims, &g);
            if (rc) return rc;
            B2_REQUIRE(job.filters && job.planes && ((uintptr_t)job.planes & 127) == 0 && (job.pass == 0 || job.pass == 1),
                       "bad argument");
            B2_REQUIRE(conv_goes_staged(g, job.pass, &list[j].a), "this convolution takes no filter tiles");
            list[j].a.staged = list[j].staged = job.planes;
            list[j].filters = (const float*)job.filters;
        }
        int count = 0;
        const int rc = b2_direct_stage_filters(list, m, &count, (cudaStream_t)stream);
        if (rc) return rc;
        *launches += count;
    }
    return B2_OK;
}

extern "C" int b2_conv_f32_tiles(int32_t pass, const float* X, const void* filter_tiles, float* O, const b2_conv_dims* d,
                                 const float* bias, const float* residual, int32_t relu, const float* mask,
                                 int32_t* status, void* stream) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(X && filter_tiles && O && status && (pass == 0 || pass == 1), "bad argument");
    b2_direct_args direct;
    B2_REQUIRE(conv_goes_staged(g, pass, &direct), "this convolution takes no filter tiles");
    direct.staged = filter_tiles;
    direct.bias = bias; direct.residual = residual; direct.relu = relu ? 1 : 0; direct.mask = mask;
    return launch_direct(direct, X, nullptr, O, nullptr, 0, 0, 0, nullptr, nullptr, status, 0, (cudaStream_t)stream);
}

extern "C" int b2_conv_fprop_f32(const float* I, const float* F, float* O, const b2_conv_dims* d,
                                 void* scratch, size_t scratch_bytes, int32_t* status,
                                 void* stream) {
    return run_fprop<float, MODE_F32X3>(I, F, O, d, nullptr, 0, 0, 0, nullptr, scratch,
                                        scratch_bytes, nullptr, status, 0, (cudaStream_t)stream);
}

extern "C" int b2_conv_fprop_flex16(const int16_t* I, const int16_t* F, int16_t* O,
                                    const b2_conv_dims* d, const b2_flex_scale* table,
                                    int32_t slotI, int32_t slotF, int32_t slotO, int32_t* stats,
                                    void* scratch, size_t scratch_bytes, uint64_t* probe_out,
                                    int32_t* status, int32_t probe, void* stream) {
    B2_REQUIRE(table && slotI >= 0 && slotF >= 0 && slotO >= 0, "flex conv needs the scale table");
    B2_REQUIRE(probe ? probe_out != nullptr : stats != nullptr, "missing statistics destination");
    return run_fprop<short, MODE_FLEX16>(I, F, O, d, table, slotI, slotF, slotO, stats, scratch,
                                         scratch_bytes, (unsigned long long*)probe_out, status,
                                         probe ? 1 : 0, (cudaStream_t)stream);
}

extern "C" int b2_conv_planes_info(const b2_conv_dims* d, int32_t pass, int32_t* supported,
                                   size_t* act_plane_bytes, size_t* filter_planes_bytes) {
    ConvGeom f, g;
    int rc = geom_from(d, &f);
    if (rc) return rc;
    B2_REQUIRE(supported && act_plane_bytes && filter_planes_bytes, "null argument");
    // The planes of a strided input gradient keep the contract that they have always had -- whole tiles
    // of 128 images, room for the error tensor at the input's resolution -- although the tensor now lies
    // undilated at the front of that room; other batches reach the tile kernel through
    // b2_conv_bprop_flex16.
    const bool strided = pass == 1 && (f.str_h > 1 || f.str_w > 1);
    *supported = pass_geom(f, pass, &g) && !(strided && f.N % 128 != 0) ? 1 : 0;
    *act_plane_bytes = 0;
    *filter_planes_bytes = 0;
    if (*supported) {
        const ImplicitShape s = implicit_shape(g);
        *act_plane_bytes = s.act_plane;
        if (strided) {
            const size_t room = plane_size(f.K, f.H + 2 * f.pad_h - f.R + 1, f.W + 2 * f.pad_w - f.S + 1, f.N);
            if (room > s.act_plane) *act_plane_bytes = room;
        }
        *filter_planes_bytes = s.filt_bytes;
    }
    return B2_OK;
}

extern "C" int b2_conv_split_activations(const int16_t* X, const b2_conv_dims* d, int32_t pass,
                                         void* planes, void* stream) {
    ConvGeom f, g;
    int rc = geom_from(d, &f);
    if (rc) return rc;
    B2_REQUIRE(X && planes && pass_geom(f, pass, &g), "planes are not available for this convolution");
    return implicit_split_activations<short, MODE_FLEX16>(X, g, implicit_shape(g), planes,
                                                          (cudaStream_t)stream);
}

extern "C" int b2_conv_split_planes(const int16_t* X, int32_t c, int32_t h, int32_t w, int32_t n,
                                    void* planes, void* stream) {
    B2_REQUIRE(X && planes && c > 0 && h > 0 && w > 0 && n > 0 && ((uintptr_t)planes & 1023) == 0, "bad argument");
    return split_to_planes(X, c, h, w, n, planes, plane_size(c, h, w, n), (cudaStream_t)stream);
}

extern "C" int b2_conv_filter_planes(const int16_t* F, const b2_conv_dims* d, int32_t pass,
                                     void* planes, void* stream) {
    ConvGeom f, g;
    int rc = geom_from(d, &f);
    if (rc) return rc;
    B2_REQUIRE(F && planes && pass_geom(f, pass, &g), "planes are not available for this convolution");
    return implicit_filter_planes(F, g, implicit_shape(g), planes, (cudaStream_t)stream);
}

extern "C" int b2_conv_filter_planes_many(const b2_conv_filter_job* list, int32_t n, int32_t* launches,
                                          void* stream) {
    B2_REQUIRE(list && n > 0 && launches, "bad argument");
    *launches = 0;
    for (int i0 = 0; i0 < n; i0 += kFilterJobs) {
        FilterJobs jobs = {};
        for (int i = i0; i < n && i < i0 + kFilterJobs; ++i) {
            ConvGeom f, g;
            int rc = geom_from(&list[i].dims, &f);
            if (rc) return rc;
            B2_REQUIRE(list[i].filters && list[i].planes && pass_geom(f, list[i].pass, &g),
                       "planes are not available for this convolution");
            if ((rc = add_filter_job(&jobs, list[i].filters, g, implicit_shape(g), list[i].planes))) return rc;
        }
        int rc = run_filter_jobs(jobs, (cudaStream_t)stream);
        if (rc) return rc;
        ++*launches;
    }
    return B2_OK;
}

extern "C" int b2_conv_flex16_planes(int32_t pass, const void* act_planes,
                                     const void* filter_planes, int16_t* out,
                                     const b2_conv_dims* d, const b2_flex_scale* table,
                                     int32_t slotX, int32_t slotF, int32_t slotOut, int32_t* stats,
                                     uint64_t* probe_out, int32_t* status, int32_t probe,
                                     void* stream) {
    ConvGeom f, g;
    int rc = geom_from(d, &f);
    if (rc) return rc;
    B2_REQUIRE(act_planes && filter_planes && out && pass_geom(f, pass, &g),
               "planes are not available for this convolution");
    B2_REQUIRE(table && slotX >= 0 && slotF >= 0 && slotOut >= 0, "flex conv needs the scale table");
    B2_REQUIRE(probe ? probe_out != nullptr : stats != nullptr, "missing statistics destination");
    return implicit_tiles(act_planes, filter_planes, out, g, implicit_shape(g), table, slotX, slotF,
                          slotOut, stats, (unsigned long long*)probe_out, status, probe ? 1 : 0,
                          (cudaStream_t)stream);
}

extern "C" int b2_conv_flex16_planes_fused(int32_t pass, const void* act_planes,
                                           const void* filter_planes, int16_t* out,
                                           const b2_conv_dims* d, const b2_flex_scale* table,
                                           int32_t slotX, int32_t slotF, int32_t slotOut,
                                           const b2_conv_epilogue* epilogue, int32_t* stats,
                                           uint64_t* probe_out, int32_t* status, int32_t probe,
                                           void* stream) {
    ConvGeom f, g;
    int rc = geom_from(d, &f);
    if (rc) return rc;
    B2_REQUIRE(act_planes && filter_planes && epilogue && pass_geom(f, pass, &g),
               "planes are not available for this convolution");
    B2_REQUIRE(out || !epilogue->write_int16, "missing output tensor");
    B2_REQUIRE(table && slotX >= 0 && slotF >= 0 && slotOut >= 0, "flex conv needs the scale table");
    B2_REQUIRE(probe ? probe_out != nullptr : stats != nullptr, "missing statistics destination");
    return implicit_tiles(act_planes, filter_planes, out, g, implicit_shape(g), table, slotX, slotF,
                          slotOut, stats, (unsigned long long*)probe_out, status, probe ? 1 : 0,
                          (cudaStream_t)stream, epilogue);
}

extern "C" int b2_conv_bprop_scratch_bytes(int32_t flex, const b2_conv_dims* d, size_t* bytes) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(bytes, "null argument");
    const int mode = flex ? MODE_FLEX16 : MODE_F32X3;
    ConvGeom gb;
    b2_direct_args direct;
    *bytes = flex && pass_geom(g, 1, &gb) ? implicit_shape(gb).bytes
             : conv_goes_direct(mode, g, 1, &direct) ? 0 : bprop_shape(mode, g).bytes;
    return B2_OK;
}

extern "C" int b2_conv_bprop_f32(const float* E, const float* F, float* GI, const b2_conv_dims* d,
                                 void* scratch, size_t scratch_bytes, int32_t* status,
                                 void* stream) {
    return run_bprop<float, MODE_F32X3>(E, F, GI, d, nullptr, 0, 0, 0, nullptr, scratch,
                                        scratch_bytes, nullptr, status, 0, (cudaStream_t)stream);
}

extern "C" int b2_conv_bprop_flex16(const int16_t* E, const int16_t* F, int16_t* GI,
                                    const b2_conv_dims* d, const b2_flex_scale* table,
                                    int32_t slotE, int32_t slotF, int32_t slotGI, int32_t* stats,
                                    void* scratch, size_t scratch_bytes, uint64_t* probe_out,
                                    int32_t* status, int32_t probe, void* stream) {
    B2_REQUIRE(table && slotE >= 0 && slotF >= 0 && slotGI >= 0, "flex conv needs the scale table");
    B2_REQUIRE(probe ? probe_out != nullptr : stats != nullptr, "missing statistics destination");
    return run_bprop<short, MODE_FLEX16>(E, F, GI, d, table, slotE, slotF, slotGI, stats, scratch,
                                         scratch_bytes, (unsigned long long*)probe_out, status,
                                         probe ? 1 : 0, (cudaStream_t)stream);
}

extern "C" int b2_conv_bprop_f32_fused(const float* E, const float* F, float* GI, const b2_conv_dims* d,
                                       const float* residual, const float* mask, int32_t* status, void* stream) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(E && F && GI, "null tensor");
    b2_direct_args direct;
    B2_REQUIRE(conv_goes_direct(MODE_F32X3, g, 1, &direct), "this convolution takes no fused tail");
    direct.residual = residual; direct.mask = mask;
    return launch_direct(direct, E, F, GI, nullptr, 0, 0, 0, nullptr, nullptr, status, 0, (cudaStream_t)stream);
}

extern "C" int b2_conv_update_scratch_bytes(int32_t flex, const b2_conv_dims* d, size_t* bytes) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(bytes, "null argument");
    const int mode = flex ? MODE_FLEX16 : MODE_F32X3;
    UpdShape u;
    b2_update_f32 f32;
    const size_t direct = update_f32_scratch(mode, g, &f32);
    *bytes = update_goes_in_planes(mode, g, &u) ? update_planes_bytes(u) : direct ? direct : update_shape(mode, g).bytes;
    return B2_OK;
}

extern "C" int b2_conv_update_planes_info(const b2_conv_dims* d, int32_t* supported, size_t* workspace_bytes) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(supported && workspace_bytes, "null argument");
    const UpdShape u = update_implicit_shape(MODE_FLEX16, g);
    *supported = u.ok ? 1 : 0;
    *workspace_bytes = u.ok ? u.acc_bytes : 0;
    return B2_OK;
}

extern "C" int b2_conv_update_flex16_planes(const void* act_planes, const void* err_planes, int16_t* U,
                                            int16_t* bias_grad, const b2_conv_dims* d,
                                            const b2_flex_scale* table, int32_t slotI, int32_t slotE,
                                            int32_t slotU, int32_t slotB, int32_t* stats, void* workspace,
                                            uint64_t* probe_out, int32_t* status, int32_t probe, void* stream) {
    ConvGeom g;
    int rc = geom_from(d, &g);
    if (rc) return rc;
    B2_REQUIRE(act_planes && err_planes && U && workspace, "null tensor");
    B2_REQUIRE(table && slotI >= 0 && slotE >= 0 && slotU >= 0 && (!bias_grad || slotB >= 0),
               "flex conv needs the scale table");
    B2_REQUIRE(probe ? probe_out != nullptr : stats != nullptr, "missing statistics destination");
    const UpdShape u = update_implicit_shape(MODE_FLEX16, g);
    B2_REQUIRE(u.ok, "this filter gradient does not read planes");
    const UpdOut o = {U, bias_grad, table, slotI, slotE, slotU, slotB, stats, (unsigned long long*)probe_out,
                      status, probe ? 1 : 0};
    return run_update_planes(act_planes, err_planes, workspace, g, u, o, (cudaStream_t)stream);
}

extern "C" int b2_conv_update_f32(const float* I, const float* E, float* U, const b2_conv_dims* d,
                                  void* scratch, size_t scratch_bytes, int32_t* status,
                                  void* stream) {
    return run_update<float, MODE_F32X3>(I, E, U, d, nullptr, 0, 0, 0, nullptr, scratch,
                                         scratch_bytes, nullptr, status, 0, (cudaStream_t)stream);
}

extern "C" int b2_conv_update_flex16(const int16_t* I, const int16_t* E, int16_t* U,
                                     const b2_conv_dims* d, const b2_flex_scale* table,
                                     int32_t slotI, int32_t slotE, int32_t slotU, int32_t* stats,
                                     void* scratch, size_t scratch_bytes, uint64_t* probe_out,
                                     int32_t* status, int32_t probe, void* stream) {
    B2_REQUIRE(table && slotI >= 0 && slotE >= 0 && slotU >= 0, "flex conv needs the scale table");
    B2_REQUIRE(probe ? probe_out != nullptr : stats != nullptr, "missing statistics destination");
    return run_update<short, MODE_FLEX16>(I, E, U, d, table, slotI, slotE, slotU, stats, scratch,
                                          scratch_bytes, (unsigned long long*)probe_out, status,
                                          probe ? 1 : 0, (cudaStream_t)stream);
}

// Gradient of pooling with respect to its input, gathered per input element (consecutive threads =
// consecutive images): the windows (p, q) that contain (h, w) are visited in increasing (p, q) --
// the order in which the reference's loop adds them (ngraph/transformers/cpu/cpuengine.py:316-336).
// avg: E / (elements of the window inside the image); max: E where (h, w) is the FIRST maximum of
// the window in row-major order (np.argmax).  flex16: fp32 arithmetic on scale_E * mantissa, one
// quantisation with the result's exponent; probe: the bit pattern of max |fp32 result|.
template <typename T, bool MAX>
__global__ void __launch_bounds__(256)
pool_bprop_kernel(const T* __restrict__ E, const T* __restrict__ I, T* __restrict__ GI, int C, int H,
                  int W, int N, int P, int Q, int R, int S, int pad_h, int pad_w, int str_h,
                  int str_w, const b2_flex_scale* __restrict__ table, int slotE, int slotG,
                  int* stats, unsigned long long* probe_out, int probe) {
    after_earlier_kernels();
    const long long total = (long long)C * H * W * N;
    const bool flex = sizeof(T) == 2;
    const float sE = flex ? table[slotE].scale : 1.0f;
    const float qG = flex && !probe ? table[slotG].inv_scale : 1.0f;
    float fstat = 0.0f, fmax = 0.0f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int n = (int)(i % N);
        long long t = i / N;
        const int w = (int)(t % W); t /= W;
        const int h = (int)(t % H);
        const int c = (int)(t / H);
        // windows with p*str - pad <= h < p*str - pad + R
        int p0 = h + pad_h - R + 1;
        p0 = p0 <= 0 ? 0 : (p0 + str_h - 1) / str_h;
        int p1 = (h + pad_h) / str_h;
        if (p1 > P - 1) p1 = P - 1;
        int q0 = w + pad_w - S + 1;
        q0 = q0 <= 0 ? 0 : (q0 + str_w - 1) / str_w;
        int q1 = (w + pad_w) / str_w;
        if (q1 > Q - 1) q1 = Q - 1;
        float acc = 0.0f;
        for (int p = p0; p <= p1; ++p)
            for (int q = q0; q <= q1; ++q) {
                const int h0 = max(p * str_h - pad_h, 0), h1 = min(p * str_h - pad_h + R, H);
                const int w0 = max(q * str_w - pad_w, 0), w1 = min(q * str_w - pad_w + S, W);
                const float e = sE * (float)E[(((long long)c * P + p) * Q + q) * N + n];
                if (MAX) {
                    // is (h, w) the first maximum of the window?
                    const T mine = I[i];
                    bool first = true;
                    for (int hh = h0; hh < h1 && first; ++hh)
                        for (int ww = w0; ww < w1; ++ww) {
                            const T v = I[(((long long)c * H + hh) * W + ww) * N + n];
                            const bool before = hh < h || (hh == h && ww < w);
                            if (v > mine || (before && v == mine)) { first = false; break; }
                        }
                    if (first) acc += e;
                } else {
                    const int cnt = (h1 - h0) * (w1 - w0);
                    acc += e * (1.0f / (float)cnt);
                }
            }
        if (!flex) {
            GI[i] = (T)acc;
        } else if (probe) {
            fmax = fmaxf(fmax, fabsf(acc));
        } else {
            float v = acc * qG;
            v = (v != v) ? 0.0f : v;
            v = fminf(fmaxf(v, -32768.0f), 32767.0f);
            fstat = fmaxf(fstat, fabsf(v));
            GI[i] = (T)(__float_as_int(v + 12582912.0f) - 0x4B400000);
        }
    }
    if (flex) {
        if (probe) {
            unsigned bits = __float_as_uint(fmax);
            for (int o = 16; o > 0; o >>= 1) bits = max(bits, __shfl_xor_sync(0xffffffffu, bits, o));
            if ((threadIdx.x & 31) == 0 && bits) atomicMax(probe_out, (unsigned long long)bits);
        } else {
            int stat = (int)rintf(fstat);
            for (int o = 16; o > 0; o >>= 1) stat = max(stat, __shfl_xor_sync(0xffffffffu, stat, o));
            if ((threadIdx.x & 31) == 0 && stat) atomicMax(stats + slotG, stat);
        }
    }
}

namespace {
int run_pool(bool is_max, const void* I, void* O, int32_t flex, int32_t C, int32_t H, int32_t W,
             int32_t N, int32_t P, int32_t Q, int32_t R, int32_t S, int32_t pad_h, int32_t pad_w,
             int32_t str_h, int32_t str_w, int32_t* stats_slot, void* stream) {
    B2_REQUIRE(I && O && C > 0 && H > 0 && W > 0 && N > 0 && P > 0 && Q > 0 && R > 0 && S > 0 &&
               str_h > 0 && str_w > 0, "bad pooling argument");
    const long long total = (long long)C * P * Q * N;
    long long blocks = (total + 31) / 32;            // 32 results per block
    if (blocks > 148 * 16) blocks = 148 * 16;
    cudaStream_t st = (cudaStream_t)stream;
#define B2_POOL_LAUNCH(T, MAXV, STATS)                                                            \
    B2_CUDA((b2::launch_after(pool_kernel<T, MAXV>, dim3((unsigned)blocks), 256, 0, st, (const T*)I, (T*)O, C, H, W, \
                              N, P, Q, R, S, pad_h, pad_w, str_h, str_w, STATS)))
    if (flex) {
        if (is_max) B2_POOL_LAUNCH(short, true, stats_slot);
        else B2_POOL_LAUNCH(short, false, stats_slot);
    } else {
        if (is_max) B2_POOL_LAUNCH(float, true, nullptr);
        else B2_POOL_LAUNCH(float, false, nullptr);
    }
#undef B2_POOL_LAUNCH
    B2_CUDA(cudaGetLastError());
    return B2_OK;
}
}  // namespace

extern "C" int b2_pool_avg_fprop(const void* I, void* O, int32_t flex, int32_t C, int32_t H,
                                 int32_t W, int32_t N, int32_t P, int32_t Q, int32_t R, int32_t S,
                                 int32_t pad_h, int32_t pad_w, int32_t str_h, int32_t str_w,
                                 int32_t* stats_slot, void* stream) {
    return run_pool(false, I, O, flex, C, H, W, N, P, Q, R, S, pad_h, pad_w, str_h, str_w,
                    stats_slot, stream);
}

extern "C" int b2_pool_max_fprop(const void* I, void* O, int32_t flex, int32_t C, int32_t H,
                                 int32_t W, int32_t N, int32_t P, int32_t Q, int32_t R, int32_t S,
                                 int32_t pad_h, int32_t pad_w, int32_t str_h, int32_t str_w,
                                 int32_t* stats_slot, void* stream) {
    return run_pool(true, I, O, flex, C, H, W, N, P, Q, R, S, pad_h, pad_w, str_h, str_w,
                    stats_slot, stream);
}

extern "C" int b2_pool_bprop(const void* E, const void* I, void* GI, int32_t flex, int32_t is_max,
                             int32_t C, int32_t H, int32_t W, int32_t N, int32_t P, int32_t Q,
                             int32_t R, int32_t S, int32_t pad_h, int32_t pad_w, int32_t str_h,
                             int32_t str_w, const b2_flex_scale* table, int32_t slotE,
                             int32_t slotGI, int32_t* stats, uint64_t* probe_out, int32_t probe,
                             void* stream) {
    B2_REQUIRE(E && GI && C > 0 && H > 0 && W > 0 && N > 0 && P > 0 && Q > 0 && R > 0 && S > 0 &&
               str_h > 0 && str_w > 0, "bad pooling argument");
    B2_REQUIRE(!is_max || I, "the gradient of max pooling needs the pooled tensor");
    if (flex) {
        B2_REQUIRE(table && slotE >= 0 && slotGI >= 0, "flex pooling gradient needs the scale table");
        B2_REQUIRE(probe ? probe_out != nullptr : stats != nullptr, "missing statistics destination");
    }
    const long long total = (long long)C * H * W * N;
    long long blocks = (total + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    cudaStream_t st = (cudaStream_t)stream;
    unsigned long long* po = (unsigned long long*)probe_out;
#define B2_PB_LAUNCH(T, MAXV)                                                                       \
    B2_CUDA((b2::launch_after(pool_bprop_kernel<T, MAXV>, dim3((unsigned)blocks), 256, 0, st, (const T*)E, \
                              (const T*)I, (T*)GI, C, H, W, N, P, Q, R, S, pad_h, pad_w, str_h, str_w, table, \
                              slotE, slotGI, stats, po, probe ? 1 : 0)))
    if (flex) {
        if (is_max) B2_PB_LAUNCH(short, true);
        else B2_PB_LAUNCH(short, false);
    } else {
        if (is_max) B2_PB_LAUNCH(float, true);
        else B2_PB_LAUNCH(float, false);
    }
#undef B2_PB_LAUNCH
    B2_CUDA(cudaGetLastError());
    return B2_OK;
}

// ---- lookup table (embedding) ----------------------------------------------------------------
namespace {
// index held as fp32, or as a flex16 mantissa with its tensor's scale
template <typename T>
__device__ __forceinline__ int lut_index(const T* idx, int i, float s) {
    return (int)rintf(s * (float)idx[i]);
}

// out = lut.take(idx, axis): lut_axis 0: lut [V][F], out [n][F]; lut_axis 1: lut [F][V], out [F][n]
template <typename T>
__global__ void __launch_bounds__(256)
lut_fprop_kernel(const T* __restrict__ lut, const T* __restrict__ idx, T* __restrict__ out,
                 int lut_axis, int V, int F, int n, const b2_flex_scale* __restrict__ table,
                 int slotI) {
    const float s_idx = table ? table[slotI].scale : 1.0f;
    const long long total = (long long)n * F;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int i = lut_axis == 0 ? (int)(e / F) : (int)(e % n);
        const int f = lut_axis == 0 ? (int)(e % F) : (int)(e / n);
        const int w = lut_index(idx, i, s_idx);
        T v = (T)0;
        if (w >= 0 && w < V) v = lut_axis == 0 ? lut[(long long)w * F + f] : lut[(long long)f * V + w];
        out[e] = v;
    }
}

// dW[w] = sum of the rows of delta whose index is w, rows added in increasing position (the order
// of np.sum over the group, ngraph/transformers/cpu/cpuengine.py:425-435); pad_idx stays zero.
// One thread per element of dW; the indices are staged through shared memory 256 at a time.
template <typename T>
__global__ void __launch_bounds__(256)
lut_update_kernel(const T* __restrict__ delta, const T* __restrict__ idx, T* __restrict__ dW,
                  int lut_axis, int V, int F, int n, int pad_idx, const b2_flex_scale* table,
                  int slotD, int slotI, int slotW, int* stats, unsigned long long* probe_out,
                  int probe) {
    __shared__ int widx[256];
    const bool flex = sizeof(T) == 2;
    const float sD = flex ? table[slotD].scale : 1.0f;
    const float sI = flex ? table[slotI].scale : 1.0f;
    const float qW = flex && !probe ? table[slotW].inv_scale : 1.0f;
    const long long total = (long long)V * F;
    const long long rounds = (total + (long long)gridDim.x * 256 - 1) / ((long long)gridDim.x * 256);
    float fstat = 0.0f, fmax = 0.0f;
    for (long long r = 0; r < rounds; ++r) {
        const long long e = (r * gridDim.x + blockIdx.x) * 256 + threadIdx.x;
        const bool live = e < total;
        const int w = live ? (lut_axis == 0 ? (int)(e / F) : (int)(e % V)) : -1;
        const int f = live ? (lut_axis == 0 ? (int)(e % F) : (int)(e / V)) : 0;
        float acc = 0.0f;
        for (int base = 0; base < n; base += 256) {
            __syncthreads();
            if (base + (int)threadIdx.x < n) widx[threadIdx.x] = lut_index(idx, base + threadIdx.x, sI);
            __syncthreads();
            const int m = min(256, n - base);
            if (live && w != pad_idx)
                for (int j = 0; j < m; ++j)
                    if (widx[j] == w) {
                        const int i = base + j;
                        acc += sD * (float)(lut_axis == 0 ? delta[(long long)i * F + f]
                                                          : delta[(long long)f * n + i]);
                    }
        }
        if (!live) continue;
        if (!flex) {
            dW[e] = (T)acc;
        } else if (probe) {
            fmax = fmaxf(fmax, fabsf(acc));
        } else {
            float v = acc * qW;
            v = (v != v) ? 0.0f : v;
            v = fminf(fmaxf(v, -32768.0f), 32767.0f);
            fstat = fmaxf(fstat, fabsf(v));
            dW[e] = (T)(__float_as_int(v + 12582912.0f) - 0x4B400000);
        }
    }
    if (flex) {
        if (probe) {
            unsigned bits = __float_as_uint(fmax);
            for (int o = 16; o > 0; o >>= 1) bits = max(bits, __shfl_xor_sync(0xffffffffu, bits, o));
            if ((threadIdx.x & 31) == 0 && bits) atomicMax(probe_out, (unsigned long long)bits);
        } else {
            int stat = (int)rintf(fstat);
            for (int o = 16; o > 0; o >>= 1) stat = max(stat, __shfl_xor_sync(0xffffffffu, stat, o));
            if ((threadIdx.x & 31) == 0 && stat) atomicMax(stats + slotW, stat);
        }
    }
}
}  // namespace

extern "C" int b2_lut_fprop(const void* lut, const void* idx, void* out, int32_t flex,
                            int32_t lut_axis, int32_t V, int32_t F, int32_t n_idx,
                            const b2_flex_scale* table, int32_t slot_idx, void* stream) {
    B2_REQUIRE(lut && idx && out && V > 0 && F > 0 && n_idx > 0 && (lut_axis == 0 || lut_axis == 1),
               "bad lookup-table argument");
    B2_REQUIRE(!flex || (table && slot_idx >= 0), "flex lookup needs the scale table");
    long long blocks = ((long long)n_idx * F + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    cudaStream_t st = (cudaStream_t)stream;
    if (flex)
        lut_fprop_kernel<short><<<(unsigned)blocks, 256, 0, st>>>(
            (const short*)lut, (const short*)idx, (short*)out, lut_axis, V, F, n_idx, table, slot_idx);
    else
        lut_fprop_kernel<float><<<(unsigned)blocks, 256, 0, st>>>(
            (const float*)lut, (const float*)idx, (float*)out, lut_axis, V, F, n_idx, nullptr, 0);
    B2_CUDA(cudaGetLastError());
    return B2_OK;
}

extern "C" int b2_lut_update(const void* delta, const void* idx, void* dW, int32_t flex,
                             int32_t lut_axis, int32_t V, int32_t F, int32_t n_idx, int32_t pad_idx,
                             const b2_flex_scale* table, int32_t slot_delta, int32_t slot_idx,
                             int32_t slot_dW, int32_t* stats, uint64_t* probe_out, int32_t probe,
                             void* stream) {
    B2_REQUIRE(delta && idx && dW && V > 0 && F > 0 && n_idx > 0 && (lut_axis == 0 || lut_axis == 1),
               "bad lookup-table argument");
    if (flex) {
        B2_REQUIRE(table && slot_delta >= 0 && slot_idx >= 0 && slot_dW >= 0,
                   "flex lookup update needs the scale table");
        B2_REQUIRE(probe ? probe_out != nullptr : stats != nullptr, "missing statistics destination");
    }
    long long blocks = ((long long)V * F + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    cudaStream_t st = (cudaStream_t)stream;
    unsigned long long* po = (unsigned long long*)probe_out;
    if (flex)
        lut_update_kernel<short><<<(unsigned)blocks, 256, 0, st>>>(
            (const short*)delta, (const short*)idx, (short*)dW, lut_axis, V, F, n_idx, pad_idx, table,
            slot_delta, slot_idx, slot_dW, stats, po, probe ? 1 : 0);
    else
        lut_update_kernel<float><<<(unsigned)blocks, 256, 0, st>>>(
            (const float*)delta, (const float*)idx, (float*)dW, lut_axis, V, F, n_idx, pad_idx, nullptr,
            0, 0, 0, nullptr, nullptr, 0);
    B2_CUDA(cudaGetLastError());
    return B2_OK;
}
