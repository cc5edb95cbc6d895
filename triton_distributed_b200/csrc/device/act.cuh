// Activations of the GEMM epilogues, on the fp32 accumulator.
#pragma once
#include <cuda_runtime.h>

#include "../include/tdist.h"

namespace tdist {

// GELU (tanh form) and SiLU are both v * sigmoid(z): one exponential and one division, and no cancellation where
// 1 + tanh(z / 2) of the textbook form has one. Their relative error grows with the argument of the exponential: z is
// rounded, __expf is good to 2 + 1.173 |z| ulps and the fast division to 2, in all below (5 + 1.2 |z|) 2^-23 for SiLU and
// (5 + 3.2 |z|) 2^-23 for GELU: 3e-5 at z = -80, where rounding to 16 bits is good to 2^-8 or 2^-11. Below z = -87.3 the divisor
// leaves the fast division's range and the result is 0, where 1.1e-36 would be the most; subnormal results are flushed.
// Measured over all finite values with results above 1e-30 (bf16) and 6e-5 (fp16): largest relative error 3.9e-3 and 4.9e-4,
// torch's SiLU the same. (Two special-function results per value: in the epilogue of a 256 x 512 tile, most of which is
// exposed, that costs more than a separate pass over the result: m2048, 4096 -> 14336 -> 4096 with GELU 443 us fused, 428 us
// apart. So only the epilogues of memory-bound tiles apply them.)
__device__ __forceinline__ float activate(float v, int act) {
    if (act == TDIST_ACT_RELU) {
        // on the bits: a float comparison would flush subnormals (--use_fast_math), and bf16 has those of fp32. NaN stays NaN.
        const uint32_t bits = __float_as_uint(v);
        return bits > 0x80000000u && bits <= 0xff800000u ? 0.f : v;
    }
    const float z = act == TDIST_ACT_GELU ? 1.5957691216057308f * v * (1.f + 0.044715f * v * v) : v;
    return v / (1.f + __expf(-z));
}
template <int N>
__device__ __forceinline__ void activate(uint32_t (&r)[N], int act) {
#pragma unroll
    for (int i = 0; i < N; ++i) r[i] = __float_as_uint(activate(__uint_as_float(r[i]), act));
}

}  // namespace tdist
