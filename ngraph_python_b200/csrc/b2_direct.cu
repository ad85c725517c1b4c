// Dispatch of the kernel with operands converted on the way in; the fp32 half of it.
#include "b2_direct.cuh"

__attribute__((visibility("hidden"))) int b2_direct_launch_flex(const b2_direct_args& a, cudaStream_t st);

long long b2_direct_cost(const b2_direct_args& a) {
    if (a.a_kind == B2_OPERAND_GATHER) {
        const b2_gather& g = a.g;
        const long long elems = (long long)g.channels * g.H * g.W * g.N;
        if (g.R * g.S > 31 || a.K > kDirMaxK || elems >= (1LL << 31)) return -1;
    }
    if ((long long)(a.M + 127) / 128 > 65535) return -1;           // grid.y
    return a.flex ? direct_shape<MODE_FLEX16>(a).cost : direct_shape<MODE_F32X3>(a).cost;
}

void b2_direct_plan(const b2_direct_args& a, b2_gemm_plan_info* plan) {
    const DirectShape s = a.flex ? direct_shape<MODE_FLEX16>(a) : direct_shape<MODE_F32X3>(a);
    *plan = {B2_GEMM_DIRECT, s.bn, s.splits, s.waves};
}

int b2_direct_launch(const b2_direct_args& a, cudaStream_t st) {
    B2_REQUIRE(b2_direct_cost(a) >= 0, "problem outside the kernel's range");
    return a.flex ? b2_direct_launch_flex(a, st) : direct_launch_mode<MODE_F32X3>(a, st);
}
