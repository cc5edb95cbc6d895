// Activation of a GEMM's result in place, for the results whose epilogue does not apply it (device/act.cuh says why).
//
// Bound by the trip of the values: the GEMM has just written them, so up to the size of L2 they are read and written there,
// which a pass into a second buffer gives away. Two special-function results per value (device/act.cuh) come second: 13 us
// for 2048 x 14336. Four 16-byte vectors per thread, loaded before the first is used. 2048 x 14336 bf16, GELU: 29 us as
// torch's pass into a new tensor; with the GEMMs before and after it (2048 x 4096 -> 14336 -> 4096) 414 us then, 401 us here.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "../device/act.cuh"
#include "../device/ptx.cuh"
#include "../include/tdist.h"
#include "../runtime/host_common.h"

namespace tdist {

constexpr int kActThreads = 256, kActVecs = 4;

template <bool F16>
__global__ void __launch_bounds__(kActThreads) activate_kernel(uint4* h, long long vecs, int act) {
    pdl_wait_and_release();
    const long long v0 = static_cast<long long>(blockIdx.x) * (kActThreads * kActVecs) + threadIdx.x;
    uint4 q[kActVecs];
#pragma unroll
    for (int u = 0; u < kActVecs; ++u)
        if (v0 + u * kActThreads < vecs) q[u] = h[v0 + u * kActThreads];
#pragma unroll
    for (int u = 0; u < kActVecs; ++u) {
        if (v0 + u * kActThreads >= vecs) break;
        uint32_t w[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float lo, hi;
            if (F16) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                lo = f.x;
                hi = f.y;
            } else {
                lo = __uint_as_float(w[i] << 16);
                hi = __uint_as_float(w[i] & 0xffff0000u);
            }
            lo = activate(lo, act);
            hi = activate(hi, act);
            w[i] = F16 ? pack_f16x2(lo, hi) : pack_bf16x2(lo, hi);
        }
        h[v0 + u * kActThreads] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

}  // namespace tdist

using namespace tdist;
using tdist_host::fail;

extern "C" int tdist_activate(void* h, long long n, int dtype, int act, void* stream) {
    if (act <= TDIST_ACT_NONE || act > TDIST_ACT_RELU) return fail(TDIST_EINVAL, "activate: unknown activation");
    if (dtype != TDIST_BF16 && dtype != TDIST_F16) return fail(TDIST_EINVAL, "activate: dtype must be bf16 or fp16");
    if (n < 0 || n % 8 || reinterpret_cast<uintptr_t>(h) % 16) return fail(TDIST_EINVAL, "activate: whole 16-byte vectors only");
    if (n == 0) return 0;
    const long long vecs = n / 8;
    const long long ctas = (vecs + kActThreads * kActVecs - 1) / (kActThreads * kActVecs);
    if (ctas > 0x7fffffffLL) return fail(TDIST_ELIMIT, "activate: too many values for one launch");
    const dim3 grid(static_cast<unsigned>(ctas));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == TDIST_F16) {
        TDIST_CUDA_OK(tdist_host::launch_pdl(activate_kernel<true>, grid, kActThreads, 0, s, static_cast<uint4*>(h), vecs, act));
    } else {
        TDIST_CUDA_OK(tdist_host::launch_pdl(activate_kernel<false>, grid, kActThreads, 0, s, static_cast<uint4*>(h), vecs, act));
    }
    return 0;
}
