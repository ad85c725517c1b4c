// The flex16 half of the kernel with operands converted on the way in.
#include "b2_direct.cuh"

__attribute__((visibility("hidden"))) int b2_direct_launch_flex(const b2_direct_args& a, cudaStream_t st) {
    return direct_launch_mode<MODE_FLEX16>(a, st);
}
