// Dispatch of the one-launch product (b2_stream.cuh); the fp32 half of it.
#include "b2_stream.cuh"

__attribute__((visibility("hidden"))) int b2_stream_launch_flex(const b2_direct_args& a, cudaStream_t st);

bool b2_product_even(const b2_direct_args& a) {
    const int size = a.flex ? 2 : 4;
    return str_even(nullptr, a.a_kind, a.a_rs, a.a_ks, size) && str_even(nullptr, a.b_kind, a.b_rs, a.b_ks, size);
}

long long b2_stream_cost(b2_direct_args& a) {
    const StreamShape s = a.flex ? stream_shape<MODE_FLEX16>(a) : stream_shape<MODE_F32X3>(a);
    a.stream = {s.bn, s.splits, s.kb_per_split, s.waves};
    return s.cost;
}

int b2_stream_launch(const b2_direct_args& a, cudaStream_t st) {
    return a.flex ? b2_stream_launch_flex(a, st) : stream_launch_mode<MODE_F32X3>(a, st);
}
