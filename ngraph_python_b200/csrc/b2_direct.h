// Launcher of the tensor-core kernel that converts its operands on the way in (b2_direct.cuh), shared
// by the GEMM and convolution entry points.  Internal to the library.
#ifndef B2_DIRECT_H
#define B2_DIRECT_H
#include "b2_common.h"

// how an operand lies: K contiguous; rows contiguous; rows gathered from a C,H,W,N tensor
enum { B2_OPERAND_K = 0, B2_OPERAND_ROWS = 1, B2_OPERAND_GATHER = 2 };

// Rows (p, q, n) of a convolution's unrolled input, or (h, w, n) of its error tensor: the value of
// column k is x[base(row) + offset(k)] where tap(k) lies inside for that row, else zero.
struct b2_gather {
    int channels, H, W, N;           // the tensor read
    int P, Q;                        // rows: pixel (p, q) of N images
    int R, S, pad_h, pad_w, str_h, str_w, dil_h, dil_w;
    int bprop;                       // columns (r, s, channel) of an input gradient, else (channel, r, s)
};

struct b2_direct_args {
    int flex;
    int a_kind, b_kind;
    const void *A, *B;
    long long a_rs, a_ks, b_rs, b_ks;   // element strides: A[row * a_rs + k * a_ks]; rows of B are columns of C
    int M, N, K;
    b2_gather g;
    void* C;
    long long ldc;
    int colmajor;                    // C[col * ldc + row] instead of C[row * ldc + col]
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

// Estimated cycles of a launch, negative where the kernel does not take the problem.
__attribute__((visibility("hidden"))) long long b2_direct_cost(const b2_direct_args& a);
__attribute__((visibility("hidden"))) int b2_direct_launch(const b2_direct_args& a, cudaStream_t st);

// fp32 filter gradient (b2_conv_update_f32.cu): no dilation, one depth.  Scratch 0: not taken.
struct b2_update_f32 { int C, H, W, N, K, R, S, P, Q, pad_h, pad_w, str_h, str_w; };
__attribute__((visibility("hidden"))) size_t b2_update_f32_scratch(const b2_update_f32& g);
__attribute__((visibility("hidden"))) int b2_update_f32_launch(const b2_update_f32& g, const float* I, const float* E,
                                                               float* U, void* scratch, int* status, cudaStream_t st);
#endif  // B2_DIRECT_H
