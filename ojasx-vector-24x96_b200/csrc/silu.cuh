// SiLU of the reference (split_manifold_lut_experiment/native/src/ojasx_lut_cpu.cpp:209-211), one rounding per operation.
#pragma once

namespace ojx {

// silu(v) = v / (1 + exp(-v))  (ojasx_lut_cpu.cpp:209-211).  exp is evaluated in double and
// rounded once, which reproduces a correctly rounded expf in all but ~1e-9 of arguments.
__device__ __forceinline__ float silu_ref(float v) {
    const float e = (float)exp((double)(-v));
    return __fdiv_rn(v, __fadd_rn(1.0f, e));
}

}  // namespace ojx
