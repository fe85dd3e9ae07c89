// dnni_span.cu -- TEST INFRASTRUCTURE: the span path's row half-widths on the
// device, for tests/test_gpu_edges.py.
#include <cstdint>

#include "../../include/dnni.h"
#include "../../terranni_b200/csrc/dnni_plan.h"

using namespace dnni;

// out[k] = half-width of the row at dy of a disc of squared radius (n0 + k * step) + dy^2.
__global__ void k_half_widths(int64_t n0, int64_t step, int dy, int n, int* out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const SpanRows r((int)(n0 + k * step + (int64_t)dy * dy), dy, dy, 1, 0, 1);
    out[k] = r.half_width();
}

extern "C" int span_half_widths(int64_t n0, int64_t step, int32_t dy, int32_t n, int32_t* out) {
    int* d = nullptr;
    if (cudaMalloc(&d, sizeof(int) * (size_t)n) != cudaSuccess) return 1;
    k_half_widths<<<(n + 255) / 256, 256>>>(n0, step, dy, n, d);
    const cudaError_t e = cudaMemcpy(out, d, sizeof(int) * (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e != cudaSuccess;
}
