// The device functions of csrc/fix64.cuh, csrc/fix64_math.cuh and their users, element by element, for tests/test_gpu_device_math.py.
// One launch evaluates function `op` for n elements: operands in a and b (bit patterns of
// doubles, or of floats in the low words; 64-bit mantissas with their exponent), the result's
// bits in out.
#include "interact32.cuh"
#include "mlp_warp.cuh"
#include "physics.cuh"

namespace sphfem {
namespace {

enum Op {
    kFixDouble, kFixScale, kFixDiv, kDiv, kFixAtan2, kAtan2, kFixSin, kFixCos, kSin, kCos, kFixPow, kPow, kFixLog, kLog,
    kPowOrLogPow, kPowOrLogLog, kRhoInv2, kRhoVol, kRhoSound, kFloatTrunc, kFloatOfNormal, kCand64, kCand32, kCandFar,
    kCandRowDiff
};

__device__ RhoTerms rho_terms_of(double rho, double mass, double bulk) {
    KConsts K{};
    K.c.phys.mass = mass;
    K.c.phys.K = bulk;
    return rho_terms(K, rho);
}
__device__ uint64_t pair_bits(float2 v) { return ((uint64_t)__float_as_uint(v.y) << 32) | __float_as_uint(v.x); }

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
        case kFixPow: return (uint64_t)__double_as_longlong(fix_pow(x, y));
        case kPow: return (uint64_t)__double_as_longlong(pow(x, y));
        case kFixLog: return (uint64_t)__double_as_longlong(fix_log_above_1(x));
        case kLog: return (uint64_t)__double_as_longlong(log(x));
        case kPowOrLogPow: return (uint64_t)__double_as_longlong(fix_pow_or_log(x, y, false));
        case kPowOrLogLog: return (uint64_t)__double_as_longlong(fix_pow_or_log(x, y, true));
        case kRhoInv2: return (uint64_t)__double_as_longlong(rho_terms_of(x, y, 1.).inv2);
        case kRhoVol: return (uint64_t)__double_as_longlong(rho_terms_of(x, y, 1.).vol);
        case kRhoSound: return (uint64_t)__double_as_longlong(rho_terms_of(x, 1., y).c);
        case kFloatTrunc: return __float_as_uint(float_trunc(x));
        case kFloatOfNormal: return __float_as_uint(float_of_normal(x));
        // a: x, y in the low and high words; b: the cell's edge; e: flags and row
        case kCand64: return pair_bits(cand_pack64(xf, __uint_as_float((uint32_t)(a >> 32)), yf, e));
        case kCand32: return pair_bits(cand_pack32(xf, __uint_as_float((uint32_t)(a >> 32)), e, yf));
        case kCandFar: return (uint32_t)cand_far(xf, __uint_as_float((uint32_t)(a >> 32)), yf);
        case kCandRowDiff: return (uint64_t)(long long)cand_row_diff(e, xf);
    }
    return 0;
}

__global__ void k_evaluate(int op, int n, const uint64_t *a, const uint64_t *b, const int *e, uint64_t *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = evaluate(op, a[i], b[i], e[i]);
}

// Counts of the floats x in [1, inf) at which recip_ge1(x) is not 1.f / x: below 2^126, and from there on
// those more than one unit off.
__global__ void k_recip_differs(unsigned long long *counts) {
    const uint32_t stride = gridDim.x * blockDim.x;
    unsigned long long differ = 0, far = 0;
    for (uint32_t b = 0x3f800000u + blockIdx.x * blockDim.x + threadIdx.x; b < 0x7f800000u; b += stride) {
        const float x = __uint_as_float(b);
        const int d = __float_as_int(recip_ge1(x)) - __float_as_int(__frcp_rn(x));
        if (x < 0x1p126f) differ += d != 0;
        else far += d < -1 || d > 1;
    }
    atomicAdd(counts, differ);
    atomicAdd(counts + 1, far);
}
__global__ void k_recip_ends(float *out) {
    out[0] = recip_ge1(__int_as_float(0x7f800000));
    out[1] = recip_ge1(__int_as_float(0x7fffffff));
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

extern "C" int device_recip(unsigned long long *counts, float *ends) {
    unsigned long long *buf = nullptr;
    cudaError_t r = cudaMalloc(&buf, 32);
    if (r == cudaSuccess) r = cudaMemset(buf, 0, 32);
    if (r == cudaSuccess) {
        sphfem::k_recip_differs<<<1216, 256>>>(buf);
        sphfem::k_recip_ends<<<1, 1>>>((float *)(buf + 2));
        r = cudaGetLastError();
    }
    if (r == cudaSuccess) r = cudaMemcpy(counts, buf, 16, cudaMemcpyDeviceToHost);
    if (r == cudaSuccess) r = cudaMemcpy(ends, buf + 2, 8, cudaMemcpyDeviceToHost);
    cudaFree(buf);
    return (int)r;
}
