// Host-side helpers shared by the launchers: error reporting, driver entry points fetched at
// run time (the library does not link libcuda), and a cache of encoded TMA descriptors.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

namespace tdist_host {

void set_error(const std::string& msg);
int fail(int code, const std::string& msg);

#define TDIST_CUDA_OK(expr)                                                              \
    do {                                                                                 \
        cudaError_t _e = (expr);                                                         \
        if (_e != cudaSuccess)                                                           \
            return ::tdist_host::fail(static_cast<int>(_e),                              \
                                      std::string(#expr) + ": " + cudaGetErrorString(_e)); \
    } while (0)

// Returns nullptr (and records an error) if the driver does not export `name`.
void* driver_fn(const char* name);

enum class Swizzle { None, B128 };

// Encodes (or fetches from the cache) a tiled tensor map of rank 2 or 3. dims/box are in
// elements, innermost first; strides_bytes[i] is the byte stride of dimension i+1.
// Returns 0 or a TDIST_E* code.
int encode_tmap(CUtensorMap* out, CUtensorMapDataType dtype, int elem_bytes, int rank_, const void* base,
                const uint64_t* dims, const uint64_t* strides_bytes, const uint32_t* box, Swizzle sw);

int sm_count();

// Launch attribute of kernels that call pdl_wait_and_release(): the grid may be set up while the stream's previous kernel
// finishes. Per pass in a row of passes: few-row GEMM m16 n6144 k12288 30.7 -> 27.2 us, gate + dispatch + dequantise +
// combine of 128 tokens 39.0 -> 35.8 us, batch-1 decode 13.2 -> 12.6 us. Not for the fp8 GEMM and its quantiser (282 -> 291 us).
inline cudaLaunchAttribute pdl_attribute() {
    cudaLaunchAttribute a;
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    return a;
}

// <<<grid, threads, smem, stream>>> with that attribute.
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, int threads, int smem, cudaStream_t stream, A... args) {
    cudaLaunchAttribute attr[1] = {pdl_attribute()};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = static_cast<size_t>(smem);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace tdist_host
