// The device functions of csrc/fix64.cuh and csrc/fix64_math.cuh, element by element, for tests/test_gpu_device_math.py.
// One launch evaluates function `op` for n elements: operands in a and b (bit patterns of
// doubles, or of floats in the low words; 64-bit mantissas with their exponent), the result's
// bits in out.
#include "physics.cuh"

namespace sphfem {
namespace {

enum Op { kFixDouble, kFixScale, kFixDiv, kDiv, kFixAtan2, kAtan2, kFixSin, kFixCos, kSin, kCos };

__device__ uint64_t evaluate(int op, uint64_t a, uint64_t b, int e) {
    const double x = __longlong_as_double((long long)a), y = __longlong_as_double((long long)b);
    const float xf = __uint_as_float((uint32_t)a), yf = __uint_as_float((uint32_t)b);
    float sn, cs;
    switch (op) {
        case kFixDouble: return (uint64_t)__double_as_longlong(fix_double({a, e}));
        case kFixScale: return (uint64_t)__double_as_longlong(fix_scale({a, e}, y, (e & 1) != 0));
        case kFixDiv: return (uint64_t)__double_as_longlong(fix_div(x, y));
        case kDiv: return (uint64_t)__double_as_longlong(x / y);
        case kFixAtan2: return __float_as_uint(fix_atan2f(yf, xf));
        case kAtan2: return __float_as_uint((float)atan2((double)yf, (double)xf));
        case kFixSin: fix_sincosf(xf, sn, cs); return __float_as_uint(sn);
        case kFixCos: fix_sincosf(xf, sn, cs); return __float_as_uint(cs);
        case kSin: return __float_as_uint((float)sin((double)xf));
        case kCos: return __float_as_uint((float)cos((double)xf));
    }
    return 0;
}

__global__ void k_evaluate(int op, int n, const uint64_t *a, const uint64_t *b, const int *e, uint64_t *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = evaluate(op, a[i], b[i], e[i]);
}

}  // namespace
}  // namespace sphfem

// Host arrays of n elements; returns the CUDA error code.
extern "C" int device_math(int op, int n, const uint64_t *a, const uint64_t *b, const int *e, uint64_t *out) {
    uint64_t *buf = nullptr;
    int *buf_e = nullptr;
    cudaError_t r = cudaMalloc(&buf, sizeof(uint64_t) * 3 * (size_t)n);
    if (r == cudaSuccess) r = cudaMalloc(&buf_e, sizeof(int) * (size_t)n);
    if (r == cudaSuccess) r = cudaMemcpy(buf, a, sizeof(uint64_t) * n, cudaMemcpyHostToDevice);
    if (r == cudaSuccess) r = cudaMemcpy(buf + n, b, sizeof(uint64_t) * n, cudaMemcpyHostToDevice);
    if (r == cudaSuccess) r = cudaMemcpy(buf_e, e, sizeof(int) * n, cudaMemcpyHostToDevice);
    if (r == cudaSuccess) {
        sphfem::k_evaluate<<<(n + 255) / 256, 256>>>(op, n, buf, buf + n, buf_e, buf + 2 * (size_t)n);
        r = cudaGetLastError();
    }
    if (r == cudaSuccess) r = cudaMemcpy(out, buf + 2 * (size_t)n, sizeof(uint64_t) * n, cudaMemcpyDeviceToHost);
    cudaFree(buf);
    cudaFree(buf_e);
    return (int)r;
}
