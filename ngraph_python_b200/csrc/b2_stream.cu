// Dispatch of the one-launch product (b2_stream.cuh); the fp32 half of it.
#include "b2_stream.cuh"

__attribute__((visibility("hidden"))) int b2_stream_launch_flex(const b2_direct_args& a, cudaStream_t st);

// Which of the two one-launch kernels a product takes.  Measured side by side on one B200, 175 sizes:
//   flex16: this one, 1.36 times as fast (geometric mean: short chains at the end, sixteen bytes to a load whatever the
//     alignment), but for one k-block and many results, where the other's two CTAs an SM hide the epilogue
//     (2929 x 567 x 122 16.1 against 23.0 us, 6714 x 264 x 86 11.4 and 15.2; 597 x 1082 x 17 18.8 and 11.5), sooner
//     where one operand only lies along K, which suits its loads (121 x 3782 x 41 7.7 and 9.3).
//   fp32: this one where the k-blocks are many enough to pay for its longer start (4: 512 x 784 x 128 5.6 against 5.9;
//     16: 512 x 128 x 512 10.7 and 8.6, transposed 13.6 and 10.0) and no line has to be shifted out of words that its
//     neighbour shares: all lines on sixteen bytes, or both operands by columns (105 x 319 x 232 9.1 and 7.7; by rows
//     99 x 1347 x 2389 17.0 and 19.3); up to two chains, or several to a CTA under a narrow result (1024 x 512 x 2048
//     22.1 and 24.3).
bool b2_product_streams(const b2_direct_args& a) {
    if (a.flex) return a.K > 128 || (long long)a.M * a.N < (a.a_kind == a.b_kind ? 900000 : 400000);
    if (a.K <= 128 || (a.K > 1024 && a.M > 32 && a.N > 32)) return false;
    return (a.a_kind == B2_OPERAND_ROWS && a.b_kind == B2_OPERAND_ROWS) ||
           (str_even(nullptr, a.a_kind, a.a_rs, a.a_ks, 4) && str_even(nullptr, a.b_kind, a.b_rs, a.b_ks, 4));
}

static StreamShape shape_of(const b2_direct_args& a) {
    return a.flex ? stream_shape<MODE_FLEX16>(a) : stream_shape<MODE_F32X3>(a);
}

long long b2_stream_cost(const b2_direct_args& a) { return shape_of(a).cost; }

void b2_stream_plan(const b2_direct_args& a, b2_gemm_plan_info* plan) {
    const StreamShape s = shape_of(a);
    *plan = {B2_GEMM_DIRECT, s.bn, s.splits, s.waves};
}

int b2_stream_launch(const b2_direct_args& a, cudaStream_t st) {
    return a.flex ? b2_stream_launch_flex(a, st) : stream_launch_mode<MODE_F32X3>(a, st);
}
