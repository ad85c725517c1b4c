// The flex16 half of the one-launch product.
#include "b2_stream.cuh"

__attribute__((visibility("hidden"))) int b2_stream_launch_flex(const b2_direct_args& a, cudaStream_t st) {
    return stream_launch_mode<MODE_FLEX16>(a, st);
}
