// sigmoid(x) in fp32 with CUDA's accurate exponential and an IEEE division: what torch.sigmoid
// computes, bit for bit wherever exp(-x) is a normal number.  --use_fast_math replaces expf, so a
// unit that includes this is built without it (build.py, ACCURATE).
#pragma once
#ifdef __USE_FAST_MATH__
#error "sigmoid.cuh: build this unit without --use_fast_math"
#endif
#include <cuda_runtime.h>

namespace ceo {

__device__ __forceinline__ float sigmoid_f32(float x) { return __fdiv_rn(1.f, 1.f + expf(-x)); }

}  // namespace ceo
