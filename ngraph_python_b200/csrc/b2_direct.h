// Launcher of the tensor-core kernel that converts its operands on the way in (b2_direct.cuh), shared
// by the GEMM and convolution entry points.  Internal to the library.
#ifndef B2_DIRECT_H
#define B2_DIRECT_H
#include "b2_common.h"

// how an operand lies: K contiguous; rows contiguous; rows gathered from a C,H,W,N tensor; rows of
// filters as the pixels of a tile see them
enum { B2_OPERAND_K = 0, B2_OPERAND_ROWS = 1, B2_OPERAND_GATHER = 2, B2_OPERAND_FILTER = 3 };

// Rows (tile, n) of a convolution: a tile is gh x gw pixels of the result and sees a window of R x S taps
// of the tensor read, tap (th, tw) at (tile_p * step_h + off_h + th * tap_h, ...).  Columns (channel,
// th, tw), or (th, tw, channel): the value there, or zero outside the tensor.
struct b2_gather {
    int channels, H, W, N;           // the tensor read
    int P, Q;                        // tiles
    int R, S, off_h, off_w, step_h, step_w, tap_h, tap_w;
    int channel_last;                // order of the columns
    // tiles of several pixels: column g * kt + k of the result is channel k of pixel g (kt a multiple of
    // 8), the result is [kt][out_p][out_q][N]; its filter row has at tap (th, tw) the filter's tap
    // r = f0_h + f1_h * th + f2_h * gy (s likewise) where that lies inside fr x fs, else zero.
    int gh, gw, kt, out_p, out_q;
    int fr, fs, f0_h, f0_w, f1_h, f1_w, f2_h, f2_w;
};

struct b2_direct_args {
    int flex;
    int a_kind, b_kind;
    const void *A, *B;
    // gathered fp32 rows: B's k-blocks as the kernel's stages hold them (b2_direct_stage_filters), or NULL
    const void* staged;
    int staged_own;                  // ... for the kernel of b2_direct.cuh, whatever b2_gather.cu makes of it
    // Gathered fp32 rows: the most k-blocks that may go into one sum (0: any).  The tensor core's sum loses
    // bits with every one, and a cheaper shape is not to lose more than callers of a layer have had: the bound
    // is what the shape of one group of producers and one pair of sums, filters as they lie, adds up in one go
    // (b2_direct_longest).
    int longest;
    long long a_rs, a_ks, b_rs, b_ks;   // element strides: A[row * a_rs + k * a_ks]; rows of B are columns of C
    int M, N, K;
    b2_gather g;
    void* C;
    long long ldc;
    int colmajor;                    // C[col * ldc + row] instead of C[row * ldc + col]
    int streams;                     // matrix products: for the kernel of b2_stream.cuh, in the shape that its cost is of
    struct { int bn, splits, kb_per_split, waves; } stream;
    const b2_flex_scale* table;
    int slotA, slotB, slotC;
    int* stats;
    unsigned long long* probe_out;
    int* status;
    int probe;
    // tail, fp32: y = relu?(product + bias[col] + residual), then 0 where mask (given) is not positive;
    // residual and mask laid out as C
    int relu;
    const float *bias, *residual, *mask;
};

// CTAs that the machine holds at once in clusters of 1..8 CTAs with an SM each (what
// cudaOccupancyMaxActiveClusters says; a cluster does not cross a GPC, and which SMs of it work differs
// from one machine to the next: 119 in clusters of seven on one, 105 on another).
constexpr int kClusterCtas[9] = {0, 148, 148, 135, 132, 130, 132, 105, 120};

// Estimated cycles of a launch, negative where the kernel does not take the problem.
__attribute__((visibility("hidden"))) long long b2_direct_cost(const b2_direct_args& a);
// The same for one group of producers and one pair of sums, and the k-blocks that then go into one sum.
__attribute__((visibility("hidden"))) long long b2_direct_longest(const b2_direct_args& a, int* longest);
// ... that do so in the shape taken.
__attribute__((visibility("hidden"))) int b2_direct_in_one_sum(const b2_direct_args& a);
// What gathered fp32 sums lose in the shape taken, in units that compare shapes and tiles of one layer and pass: every
// step of eight columns cuts a sum off below its last bit, in the same direction, so that a sum of n steps of one size
// loses about n^1.5 of what a step adds, and sums of their own add up as their squares.  Columns that a pixel does not
// see are zeros and cost nothing.  (Against 64 bits: errors of two shapes have this ratio to within 1.15, none is larger
// by more than 1.01 where this is not, 113 layers and passes.)
__attribute__((visibility("hidden"))) double b2_direct_loss(const b2_direct_args& a);
__attribute__((visibility("hidden"))) void b2_direct_plan(const b2_direct_args& a, b2_gemm_plan_info* plan);
// `staged` operands: bytes, and the kernel that makes those of n products (fewest launches; `launches`
// counts them).  Whether a product has its operand staged changes its shape, so `staged` is set (to
// anything) for b2_direct_cost, b2_direct_plan and here alike.
constexpr int kStageJobs = 16;
struct b2_stage_job { b2_direct_args a; const float* filters; void* staged; };
__attribute__((visibility("hidden"))) size_t b2_direct_staged_bytes(const b2_direct_args& a);
__attribute__((visibility("hidden"))) int b2_direct_stage_filters(const b2_stage_job* jobs, int n, int* launches,
                                                                  cudaStream_t st);
__attribute__((visibility("hidden"))) int b2_direct_launch(const b2_direct_args& a, cudaStream_t st);

// Matrix products of operands as they lie (b2_stream.cuh): likewise; whether all lines of both start on sixteen bytes
// if the operands do.
__attribute__((visibility("hidden"))) bool b2_product_even(const b2_direct_args& a);
__attribute__((visibility("hidden"))) long long b2_stream_cost(b2_direct_args& a);            // (sets a.stream)
__attribute__((visibility("hidden"))) int b2_stream_launch(const b2_direct_args& a, cudaStream_t st);

// Gathered products whose filters are laid out beforehand (b2_gather.cu): whether it takes one rather than the kernel
// above, its cost and shape (tile, slices, waves, k-blocks in one sum of large terms and in one of small ones), and the
// launch.  K-block n has its planes in the other order where `turned` is not 0 and n / turned odd.
struct b2_gather_info { long long cost; int bn, splits, waves, kb_per_split, sums, in_one_sum, small, turned; };
__attribute__((visibility("hidden"))) bool b2_gather_streams(const b2_direct_args& a);
__attribute__((visibility("hidden"))) b2_gather_info b2_gather_plan(const b2_direct_args& a);
__attribute__((visibility("hidden"))) int b2_gather_launch(const b2_direct_args& a, cudaStream_t st);

// fp32 filter gradient (b2_conv_update_f32.cu): no dilation, one depth.  Scratch 0: not taken.
struct b2_update_f32 { int C, H, W, N, K, R, S, P, Q, pad_h, pad_w, str_h, str_w; };
__attribute__((visibility("hidden"))) size_t b2_update_f32_scratch(const b2_update_f32& g);
__attribute__((visibility("hidden"))) int b2_update_f32_launches(const b2_update_f32& g);
__attribute__((visibility("hidden"))) int b2_update_f32_launch(const b2_update_f32& g, const float* I, const float* E,
                                                               float* U, void* scratch, int* status, cudaStream_t st);
#endif  // B2_DIRECT_H
