// Dispatch of the one-launch product (b2_stream.cuh); the fp32 half of it.
#include "b2_stream.cuh"

__attribute__((visibility("hidden"))) int b2_stream_launch_flex(const b2_direct_args& a, cudaStream_t st);

bool b2_product_even(const b2_direct_args& a) {
    const int size = a.flex ? 2 : 4;
    return str_even(nullptr, a.a_kind, a.a_rs, a.a_ks, size) && str_even(nullptr, a.b_kind, a.b_rs, a.b_ks, size);
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
