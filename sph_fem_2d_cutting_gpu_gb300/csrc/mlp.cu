// mlp.cu -- the learned warm start of the Johnson-Cook return mapping: a
// 4-64-64-64-1 SiLU MLP with BF16 weights and FP32 accumulation that predicts
// the plastic-multiplier increment, its training (forward, backward, Adam)
// and the warm-started return mapping of the fused FP32-compensated step.
//
// The 64x64 hidden layers run on the 5th-generation tensor cores: operands in
// shared memory in the no-swizzle K-major layout, tcgen05.mma issued by one
// thread, accumulators in TMEM, completion through tcgen05.commit on an
// mbarrier.  A tile is 128 samples = the 128 TMEM lanes of an M=128 accumulator,
// read with tcgen05.ld 32x32b: one thread for each sample in inference, four
// (16 neurons each) in training.  In training the two
// 64x64 weight gradients of a tile are one M=128, N=128, K=128 MMA
// ([dZ3^T; dZ2^T] x [A2 | A1]: the two diagonal blocks are dW3 and dW2) that
// accumulates in TMEM over all tiles of the CTA.
//
// Every wait on the tensor cores is bounded (1 s, then SPH_STATUS_MMA_TIMEOUT
// and an orderly exit that still frees TMEM).
#include <cuda_bf16.h>

#include "async.cuh"
#include "launch.cuh"
#include "mlp_warp.cuh"

namespace sphfem {
namespace {

constexpr int kTile = 128;                 // samples per tile (inference: threads per CTA)
constexpr uint32_t kTmemCols = 256;        // training: [0,64) layer, [64,192) stacked dW
constexpr uint32_t kTmemColsFwd = 64;      // inference

// Instruction descriptor of tcgen05.mma kind::f16: D F32 (bits 4-5 = 1), A and
// B BF16 (bits 7-9, 10-12 = 1), both K-major, N>>3 at bit 17, M>>4 at bit 24.
constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Byte offset of element (row r, column k) of a K-major BF16 operand with kt
// columns: 8x8 core matrices of 8 rows x 16 bytes (128 contiguous bytes);
// along K the core matrices are 128 bytes apart (leading byte offset), along
// the rows the 8-row groups are kt*16 bytes apart (stride byte offset).
__device__ __forceinline__ uint32_t cm_off(int r, int k, int kt) {
    return (uint32_t)((r >> 3) * (kt * 16) + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// Shared-memory matrix descriptor (no swizzle, version 1 at bits 46-48).
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

// D[128 x N] (+)= A[128 x kt] * B[N x kt]^T, both K-major in shared memory.
__device__ __forceinline__ void gemm_issue(uint32_t tmem_d, uint32_t a_saddr, uint32_t b_saddr, int kt, int N,
                                           bool accumulate) {
    const uint32_t sbo = (uint32_t)kt * 16;
    const uint32_t idesc = idesc_bf16(128, N);
    for (int s = 0; s < kt / 16; s++) {
        uint64_t a = sdesc(a_saddr + 256u * s, 128, sbo);
        uint64_t b = sdesc(b_saddr + 256u * s, 128, sbo);
        mma_bf16(tmem_d, a, b, idesc, (accumulate || s > 0) ? 1u : 0u);
    }
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Whole warp: allocate `ncols` TMEM columns, address written to smem slot.
__device__ __forceinline__ void tmem_alloc(uint32_t slot_saddr, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_saddr), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane (load + wait in one
// statement, so no use of the registers can be scheduled before the wait).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// d silu(z) / dz from the sigmoid s of z.
__device__ __forceinline__ float dsiluf_(float z, float s) { return s * (1.f + z * (1.f - s)); }

// Four 8x8 BF16 core matrices (128 contiguous bytes each) transposed from shared to
// shared memory by one warp; lane l passes the address of row l & 7 of matrix l >> 3.
__device__ __forceinline__ void transpose_cores(uint32_t dst, uint32_t src) {
    uint32_t a, b, c, d;
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(a), "=r"(b), "=r"(c), "=r"(d)
                 : "r"(src)
                 : "memory");
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(a), "r"(b), "r"(c),
                 "r"(d)
                 : "memory");
}

// Shared parameter block of a CTA (FP32 values of the BF16 weights of the
// CUDA-core layers, biases).
struct MlpSmall {
    float w1[kMlpH * kMlpIn], b1[kMlpH], b2[kMlpH], b3[kMlpH], w4[kMlpH], b4;
};

__device__ void load_small(MlpSmall &s, const MlpDev &m) {
    for (int i = threadIdx.x; i < kMlpH * kMlpIn; i += blockDim.x) s.w1[i] = bf16_bits_to_f(m.wb[kMlpWbW1 + i]);
    for (int i = threadIdx.x; i < kMlpH; i += blockDim.x) {
        s.b1[i] = m.params[kMlpOffB1 + i];
        s.b2[i] = m.params[kMlpOffB2 + i];
        s.b3[i] = m.params[kMlpOffB3 + i];
        s.w4[i] = bf16_bits_to_f(m.wb[kMlpWbW4 + i]);
    }
    if (threadIdx.x == 0) s.b4 = m.params[kMlpOffB4];
}

// W [64 out][64 in] as the B operand of X W^T (rows n = out, K = in): 8 consecutive
// inputs of one output are one 16-byte core-matrix row.
__device__ void load_weight(unsigned char *dst, const uint16_t *w) {
    for (int i = threadIdx.x; i < kMlpH * kMlpH / 8; i += blockDim.x) {
        const int o = i >> 3, k8 = (i & 7) * 8;
        *(uint4 *)(dst + cm_off(o, k8, 64)) = *(const uint4 *)(w + o * kMlpH + k8);
    }
}

// Shared memory of the forward-only kernels.
struct FwdSmem {
    alignas(128) unsigned char w2[kMlpH * kMlpH * 2];
    alignas(128) unsigned char w3[kMlpH * kMlpH * 2];
    alignas(128) unsigned char act[kTile * kMlpH * 2];
    MlpSmall small;
    alignas(8) unsigned long long mbar;
    uint32_t tmem_slot;
    int fail;
};

// 16 columns [c0, c0+16) of row r of a K-major 64-column operand (BF16).
__device__ __forceinline__ void store_row16(unsigned char *base, int r, int c0, const float *v) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const float *w = v + 8 * h;
        *(uint4 *)(base + cm_off(r, c0 + 8 * h, 64)) =
            make_uint4(pack_bf16x2(w[0], w[1]), pack_bf16x2(w[2], w[3]), pack_bf16x2(w[4], w[5]),
                       pack_bf16x2(w[6], w[7]));
    }
}

// Forward pass of this CTA's tile; xn = standardised features of this
// thread's row.  Returns the standardised output, or sets *timeout.  The
// activations go 16 columns at a time (TMEM load, SiLU, store) in a rolled
// loop: the code stays small enough for the instruction cache of a short,
// latency-bound launch.
// skip_mma (failure-path tests): issue no MMA, so the bounded wait runs out.
__device__ float forward_tile(FwdSmem &sh, uint32_t tmem, uint32_t &phase, const float *xn, bool &timeout,
                              bool skip_mma = false) {
    const uint32_t mbar = smem_u32(&sh.mbar);
    const int r = threadIdx.x;
    const uint32_t trow = tmem + (((uint32_t)threadIdx.x >> 5) * 32u << 16);
    float v[16];
#pragma unroll 1
    for (int c0 = 0; c0 < kMlpH; c0 += 16) {   // layer 1 on the CUDA cores
#pragma unroll
        for (int q = 0; q < 16; q++) {
            float acc = sh.small.b1[c0 + q];
#pragma unroll
            for (int c = 0; c < kMlpIn; c++) acc = fmaf(sh.small.w1[(c0 + q) * kMlpIn + c], xn[c], acc);
            v[q] = siluf_(acc);
        }
        store_row16(sh.act, r, c0, v);
    }
    float y = sh.small.b4;
#pragma unroll 1
    for (int layer = 0; layer < 2; layer++) {
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (r == 0 && !skip_mma) {
            tc_fence_after();
            gemm_issue(tmem, smem_u32(sh.act), smem_u32(layer == 0 ? sh.w2 : sh.w3), 64, 64, false);
            mma_commit(mbar);
        }
        bool ok = mbar_wait(mbar, phase);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
            timeout = true;
            return 0.f;
        }
        tc_fence_after();
        const float *b = layer == 0 ? sh.small.b2 : sh.small.b3;
#pragma unroll 1
        for (int c0 = 0; c0 < kMlpH; c0 += 16) {
            tmem_ld16(trow + c0, v);
            if (layer == 0) {   // the MMA has read act: overwrite it with A2 (next MMA after the barrier)
#pragma unroll
                for (int q = 0; q < 16; q++) v[q] = siluf_(v[q] + b[c0 + q]);
                store_row16(sh.act, r, c0, v);
            } else {
#pragma unroll
                for (int q = 0; q < 16; q++) y = fmaf(sh.small.w4[c0 + q], siluf_(v[q] + b[c0 + q]), y);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    return y;
}

__device__ bool fwd_setup(FwdSmem &sh, const MlpDev &m, uint32_t &tmem) {
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&sh.mbar));
        sh.fail = 0;
    }
    load_small(sh.small, m);
    load_weight(sh.w2, m.wb + kMlpWbW2);
    load_weight(sh.w3, m.wb + kMlpWbW3);
    if (threadIdx.x < 32) tmem_alloc(smem_u32(&sh.tmem_slot), kTmemColsFwd);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem = sh.tmem_slot;
    return true;
}

__device__ void fwd_teardown(FwdSmem &sh, uint32_t tmem) {
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemColsFwd);
    }
}

// ---- batch inference (raw features in, raw target out) -------------------------------------------
__global__ void __launch_bounds__(kTile, 1) k_mlp_predict(MlpDev m, const float *__restrict__ x, int64_t n,
                                                         float *__restrict__ y, uint32_t *status) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    FwdSmem &sh = *(FwdSmem *)smem_raw;
    const int64_t ntiles = (n + kTile - 1) / kTile;
    if ((int64_t)blockIdx.x >= ntiles) return;
    uint32_t tmem;
    fwd_setup(sh, m, tmem);
    uint32_t phase = 0;
    for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int64_t i = t * kTile + threadIdx.x;
        float xr[kMlpIn] = {0.f, 0.f, 0.f, 0.f}, xn[kMlpIn];
        if (i < n) {
            float4 q = *(const float4 *)(x + 4 * i);
            xr[0] = q.x; xr[1] = q.y; xr[2] = q.z; xr[3] = q.w;
        }
        normalise(m, xr, xn);
        bool timeout = false;
        float yh = forward_tile(sh, tmem, phase, xn, timeout);
        if (timeout) {
            if (threadIdx.x == 0) set_status(status, SPH_STATUS_MMA_TIMEOUT);
            break;
        }
        if (i < n) y[i] = yh * m.y_std + m.y_mean;
    }
    fwd_teardown(sh, tmem);
}

// ---- batch inference, 16 samples per warp pass (the fused step's in-epilogue form) -----------------
__global__ void __launch_bounds__(256) k_mlp_predict_warp(MlpDev m, const float *__restrict__ x, int64_t n,
                                                         float *__restrict__ y) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w * 16 < n; w += warps) {
        const int64_t i = w * 16 + lane;   // lanes 0..15 hold the samples (warp-uniform loop)
        const bool valid = lane < 16 && i < n;
        float xr[kMlpIn] = {0.f, 0.f, 0.f, 0.f}, xn[kMlpIn];
        if (valid) {
            const float4 q = __ldg((const float4 *)x + i);
            xr[0] = q.x; xr[1] = q.y; xr[2] = q.z; xr[3] = q.w;
        }
        normalise(m, xr, xn);
        const unsigned rows = __ballot_sync(0xffffffffu, valid);
        const float yh = mlp_forward_warp16(m, rows, xn);
        if (valid) y[i] = yh * m.y_std + m.y_mean;
    }
}

// ---- warm-started return mapping of the fused FP32 step (tensor-core form) -----------------------
__global__ void __launch_bounds__(kTile, 1)
    k_jc_warm(KConsts K, SortedFields32 B, FixedFields32 F, const ToolDev *__restrict__ tool, MlpDev m,
              int32_t *__restrict__ secant_iters, uint32_t *status) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    FwdSmem &sh = *(FwdSmem *)smem_raw;
    const int count = *K.jc_list_count;
    const int ntiles = (count + kTile - 1) / kTile;
    if ((int)blockIdx.x >= ntiles) return;
    uint32_t tmem;
    fwd_setup(sh, m, tmem);
    uint32_t phase = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int e = t * kTile + threadIdx.x;
        const bool valid = e < count;
        const int k = valid ? K.jc_list[e] : 0;
        JcWarmState st{};
        float x[kMlpIn] = {0.f, 0.f, 0.f, 0.f}, xn[kMlpIn];
        if (valid) jc_warm_load(K, B, F, k, st, x);
        normalise(m, x, xn);
        bool timeout = false;
        const float yh = forward_tile(sh, tmem, phase, xn, timeout, (K.test_faults & SPH_TEST_SKIP_MMA) != 0);
        if (timeout) {
            if (threadIdx.x == 0) set_status(status, SPH_STATUS_MMA_TIMEOUT);
            break;
        }
        if (valid) jc_warm_finish(K, B, tool, m, k, yh, st, secant_iters, status);
    }
    fwd_teardown(sh, tmem);
}

// ---- training: gradients of one minibatch ---------------------------------------------------------
constexpr int kTrainThreads = 512;   // four threads for each sample of a tile, 16 neurons each

struct TrainSmem {
    alignas(128) unsigned char w2f[kMlpH * kMlpH * 2];   // W2 as B of A1 W2^T
    alignas(128) unsigned char w3f[kMlpH * kMlpH * 2];
    alignas(128) unsigned char w2b[kMlpH * kMlpH * 2];   // W2^T as B of dZ2 W2
    alignas(128) unsigned char w3b[kMlpH * kMlpH * 2];
    alignas(128) unsigned char act[kTile * kMlpH * 2];   // A operand of the 64-wide GEMMs
    alignas(128) unsigned char adw[kTile * kTile * 2];   // [dZ3^T; dZ2^T]  (rows: neurons, K: samples)
    alignas(128) unsigned char bdw[kTile * kTile * 2];   // [A2^T; A1^T]
    float zs[kTile][kMlpH + 1];                          // A3 of each sample, then dZ1; at the end the sums to merge
    alignas(16) float xn[kTile][kMlpIn];
    float g[kTile];                                      // d loss / dy of each sample
    float db4[4], loss[4];
    MlpSmall small;
    alignas(8) unsigned long long mbar, mbar_dw;
    uint32_t tmem_slot;
};

// Per-CTA partial sums over the samples of its tiles, written to
// part[blockIdx.x][0..kMlpParams) (gradient of the mean loss) and
// part[..][kMlpParams] (sum of 0.5 (y - t)^2 in standardised units).
//
// A tile's chain is five MMAs with the SiLU of 128 x 64 values between them, so it is
// bound by the latency of that chain and by the sigmoids (three for each sample and
// neuron, each with its derivative).  With one thread for each sample the 64-wide
// register rows unrolled into code far larger than the instruction cache and one warp
// in flight on each scheduler: 50 us a tile.  Four threads for each sample (16 neurons
// each: straight-line code, four warps on each scheduler), the sigmoids evaluated once,
// the transposed operands of the weight gradient made from the stored ones by
// ldmatrix / stmatrix while the layer's MMA runs, and sums over the samples split over
// all threads: 65,536 samples (512 tiles on 152 SMs) 226 -> 48 us, and 42 us with the
// sigmoid's reciprocal free of branches; 8,192 samples 92 -> 18 us.
__global__ void __launch_bounds__(kTrainThreads, 1)
    k_mlp_grad(MlpDev m, const float *__restrict__ x, const float *__restrict__ tgt, const int32_t *__restrict__ idx,
               int64_t nb, float inv_nb, float *__restrict__ part, uint32_t *status) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    TrainSmem &sh = *(TrainSmem *)smem_raw;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = tid & (kTile - 1), c0 = 16 * (tid >> 7);   // this thread's sample (TMEM lane) and first neuron
    const int nj = tid & (kMlpH - 1), ns = 16 * (tid >> 6);  // in sums over samples: its neuron and first sample
    float *out = part + (size_t)blockIdx.x * (kMlpParams + 1);
    const int64_t ntiles = (nb + kTile - 1) / kTile;
    if ((int64_t)blockIdx.x >= ntiles) {
        for (int i = tid; i < kMlpParams + 1; i += kTrainThreads) out[i] = 0.f;
        return;
    }
    const uint32_t mbar = smem_u32(&sh.mbar), mbar_dw = smem_u32(&sh.mbar_dw);
    const uint32_t act = smem_u32(sh.act), adw = smem_u32(sh.adw), bdw = smem_u32(sh.bdw);
    if (tid == 0) {
        mbar_init(mbar);
        mbar_init(mbar_dw);
    }
    load_small(sh.small, m);
    load_weight(sh.w2f, m.wb + kMlpWbW2);
    load_weight(sh.w3f, m.wb + kMlpWbW3);
    if (warp == 0) tmem_alloc(smem_u32(&sh.tmem_slot), kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_slot;
    const uint32_t trow = tmem + ((uint32_t)(warp & 3) * 32u << 16) + (uint32_t)c0;
    {   // the transposed weights: warp w does the 8 outputs of group w / 2 and 32 inputs
        const uint32_t o = (uint32_t)(warp >> 1), i = (uint32_t)(4 * (warp & 1) + (lane >> 3)), b = 16u * (lane & 7);
        transpose_cores(smem_u32(sh.w2b) + i * 1024 + o * 128 + b, smem_u32(sh.w2f) + o * 1024 + i * 128 + b);
        transpose_cores(smem_u32(sh.w3b) + i * 1024 + o * 128 + b, smem_u32(sh.w3f) + o * 1024 + i * 128 + b);
    }
    uint32_t phase = 0, phase_dw = 0;
    bool timeout = false;
    // sums of this thread: dW1[nj][:], db1[nj], dW4[nj] over its samples; db3 / db2 of row r of
    // adw over its quarter of the samples; threads of the first 16 neurons: db4 and the loss
    float acc_w1[kMlpIn] = {0.f, 0.f, 0.f, 0.f}, acc_b1 = 0.f, acc_w4 = 0.f, acc_b23 = 0.f, acc_b4 = 0.f, acc_loss = 0.f;
    int tiles_done = 0;
    float v[16], d1[16], d2[16];

    auto mma_wait = [&](uint32_t bar, uint32_t &ph) -> bool {
        bool ok = mbar_wait(bar, ph);
        ph ^= 1u;
        const bool all = !__syncthreads_or(!ok);
        tc_fence_after();
        return all;
    };
    auto sync_for_mma = [&]() {
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
    };
    auto issue = [&](const unsigned char *w) {   // layer accumulator = act w^T
        if (tid == 0) {
            tc_fence_after();
            gemm_issue(tmem, act, smem_u32(w), 64, 64, false);
            mma_commit(mbar);
        }
    };
    // act^T (64 neurons x 128 samples) into rows row0.. of an operand of the weight gradient:
    // a warp does 8 samples
    auto transpose_act = [&](uint32_t dst, int row0) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t ng = (uint32_t)(4 * h + (lane >> 3)), b = 16u * (lane & 7);
            transpose_cores(dst + ((uint32_t)(row0 >> 3) + ng) * 2048u + (uint32_t)warp * 128u + b,
                            act + (uint32_t)warp * 1024u + ng * 128u + b);
        }
    };

    for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int64_t e = t * kTile + r;
        const bool valid = e < nb;
        float xr[kMlpIn] = {0.f, 0.f, 0.f, 0.f}, xn[kMlpIn], tn = 0.f;
        if (valid) {
            const int64_t i = idx ? idx[e] : e;
            float4 q = *(const float4 *)(x + 4 * i);
            xr[0] = q.x; xr[1] = q.y; xr[2] = q.z; xr[3] = q.w;
            if (c0 == 0) tn = (tgt[i] - m.y_mean) / m.y_std;
        }
        normalise(m, xr, xn);
        if (c0 == 0) *(float4 *)sh.xn[r] = make_float4(xn[0], xn[1], xn[2], xn[3]);
        // layer 1 (CUDA cores)
#pragma unroll
        for (int q = 0; q < 16; q++) {
            float z = sh.small.b1[c0 + q];
#pragma unroll
            for (int c = 0; c < kMlpIn; c++) z = fmaf(sh.small.w1[(c0 + q) * kMlpIn + c], xn[c], z);
            const float s = sigmoidf_(z);
            d1[q] = dsiluf_(z, s);
            v[q] = z * s;
        }
        store_row16(sh.act, r, c0, v);
        // layer 2: Z2 = A1 W2^T + b2
        sync_for_mma();
        issue(sh.w2f);
        transpose_act(bdw, 64);   // A1^T
        if (!mma_wait(mbar, phase)) { timeout = true; break; }
        tmem_ld16(trow, v);
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const float z = v[q] + sh.small.b2[c0 + q], s = sigmoidf_(z);
            d2[q] = dsiluf_(z, s);
            v[q] = z * s;
        }
        store_row16(sh.act, r, c0, v);
        // layer 3: Z3 = A2 W3^T + b3, output, dZ3
        sync_for_mma();
        issue(sh.w3f);
        transpose_act(bdw, 0);   // A2^T
        if (!mma_wait(mbar, phase)) { timeout = true; break; }
        tmem_ld16(trow, v);
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const float z = v[q] + sh.small.b3[c0 + q], s = sigmoidf_(z);
            sh.zs[r][c0 + q] = z * s;
            v[q] = dsiluf_(z, s);
        }
        __syncthreads();
        if (c0 == 0) {   // the output: one thread for each sample
            float y = sh.small.b4;
#pragma unroll 16
            for (int j = 0; j < kMlpH; j++) y = fmaf(sh.small.w4[j], sh.zs[r][j], y);
            const float err = valid ? (y - tn) : 0.f;
            const float g = err * inv_nb;
            sh.g[r] = g;
            acc_b4 += g;
            acc_loss = fmaf(0.5f * err, err, acc_loss);
        }
        __syncthreads();
        {
            const float g = sh.g[r];
#pragma unroll
            for (int q = 0; q < 16; q++) v[q] = g * sh.small.w4[c0 + q] * v[q];
        }
        store_row16(sh.act, r, c0, v);   // dZ3 as A of dA2 = dZ3 W3
        sync_for_mma();
        issue(sh.w3b);
        transpose_act(adw, 0);           // dZ3^T
#pragma unroll
        for (int s = 0; s < 16; s++) acc_w4 = fmaf(sh.g[ns + s], sh.zs[ns + s][nj], acc_w4);
        if (!mma_wait(mbar, phase)) { timeout = true; break; }
        tmem_ld16(trow, v);
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = v[q] * d2[q];
        store_row16(sh.act, r, c0, v);   // dZ2 as A of dA1 = dZ2 W2
        sync_for_mma();
        issue(sh.w2b);
        transpose_act(adw, 64);          // dZ2^T
        // [dW3 | . ; . | dW2] += [dZ3^T; dZ2^T] [A2 | A1] over this tile's samples
        sync_for_mma();
        if (tid == 0) {
            tc_fence_after();
            gemm_issue(tmem + 64, adw, bdw, 128, 128, tiles_done > 0);
            mma_commit(mbar_dw);
        }
        if (!mma_wait(mbar, phase)) {
            mbar_wait(mbar_dw, phase_dw);   // (bounded) the weight gradient in flight, before its TMEM is freed
            timeout = true;
            break;
        }
        tmem_ld16(trow, v);
#pragma unroll
        for (int q = 0; q < 16; q++) sh.zs[r][c0 + q] = v[q] * d1[q];   // dZ1 (FP32)
        tc_fence_before();
        __syncthreads();
#pragma unroll
        for (int s = 0; s < 16; s++) {
            const float d = sh.zs[ns + s][nj];
            const float4 xs = *(const float4 *)sh.xn[ns + s];
            acc_b1 += d;
            acc_w1[0] = fmaf(d, xs.x, acc_w1[0]);
            acc_w1[1] = fmaf(d, xs.y, acc_w1[1]);
            acc_w1[2] = fmaf(d, xs.z, acc_w1[2]);
            acc_w1[3] = fmaf(d, xs.w, acc_w1[3]);
        }
        {
            float sum = 0.f;
#pragma unroll
            for (int k8 = 0; k8 < 32; k8 += 8) {
                const uint4 q = *(const uint4 *)(sh.adw + cm_off(r, 2 * c0 + k8, 128));   // 2 c0: the quarter's samples
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int h = 0; h < 4; h++)
                    sum += __uint_as_float(w[h] << 16) + __uint_as_float(w[h] & 0xffff0000u);
            }
            acc_b23 += sum;
        }
        tiles_done++;
        if (!mma_wait(mbar_dw, phase_dw)) { timeout = true; break; }   // act, adw, bdw, zs free again
    }
    if (timeout) {
        if (tid == 0) set_status(status, SPH_STATUS_MMA_TIMEOUT);
        for (int i = tid; i < kMlpParams + 1; i += kTrainThreads) out[i] = 0.f;
    } else {
        // weight gradients from TMEM: rows < 64 hold dW3 (columns 64..127), rows >= 64 dW2 (columns 128..191)
        const bool upper = r < kMlpH;
        tmem_ld16(trow + (upper ? 64u : 128u), v);
        float *dst = out + (upper ? kMlpOffW3 + r * kMlpH : kMlpOffW2 + (r - kMlpH) * kMlpH) + c0;
#pragma unroll
        for (int q = 0; q < 16; q += 2) *(float2 *)(dst + q) = make_float2(v[q], v[q + 1]);
        float(&red)[7][kTrainThreads] = *(float(*)[7][kTrainThreads]) & sh.zs[0][0];
        red[0][tid] = acc_w1[0];
        red[1][tid] = acc_w1[1];
        red[2][tid] = acc_w1[2];
        red[3][tid] = acc_w1[3];
        red[4][tid] = acc_b1;
        red[5][tid] = acc_w4;
        red[6][tid] = acc_b23;
        if (c0 == 0) {
            for (int o = 16; o > 0; o >>= 1) {
                acc_b4 += __shfl_xor_sync(0xffffffffu, acc_b4, o);
                acc_loss += __shfl_xor_sync(0xffffffffu, acc_loss, o);
            }
            if (lane == 0) { sh.db4[warp] = acc_b4; sh.loss[warp] = acc_loss; }
        }
        __syncthreads();
        if (tid < 6 * kMlpH) {   // sum m of neuron nj over the 8 groups of samples
            const int mm = tid >> 6;
            float s = 0.f;
#pragma unroll
            for (int h = 0; h < 8; h++) s += red[mm][h * kMlpH + nj];
            out[mm < 4 ? kMlpOffW1 + nj * kMlpIn + mm : (mm == 4 ? kMlpOffB1 : kMlpOffW4) + nj] = s;
        } else {                 // rows nj and 64 + nj of adw over the four quarters
            const int row = tid - 6 * kMlpH;
            const float s = (red[6][row] + red[6][kTile + row]) + (red[6][2 * kTile + row] + red[6][3 * kTile + row]);
            out[(row < kMlpH ? kMlpOffB3 : kMlpOffB2 - kMlpH) + row] = s;
        }
        if (tid == 0) {
            out[kMlpOffB4] = sh.db4[0] + sh.db4[1] + sh.db4[2] + sh.db4[3];
            out[kMlpParams] = sh.loss[0] + sh.loss[1] + sh.loss[2] + sh.loss[3];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// BF16 copy of parameter p if it is a weight.
__device__ __forceinline__ void store_wb(uint16_t *__restrict__ wb, int p, float w) {
    int q = -1;
    if (p < kMlpOffB1) q = kMlpWbW1 + p;
    else if (p >= kMlpOffW2 && p < kMlpOffB2) q = kMlpWbW2 + (p - kMlpOffW2);
    else if (p >= kMlpOffW3 && p < kMlpOffB3) q = kMlpWbW3 + (p - kMlpOffW3);
    else if (p >= kMlpOffW4 && p < kMlpOffB4) q = kMlpWbW4 + (p - kMlpOffW4);
    if (q >= 0) wb[q] = __bfloat16_as_ushort(__float2bfloat16_rn(w));
}

// Sum of the per-CTA partials in a fixed order (deterministic); with `adam`, one
// Adam step on the FP32 parameters and refreshed BF16 weight copies.  A block has 32
// parameters and eight groups of CTAs: one thread for each parameter walked up to 304
// partials in turn on 35 SMs, 15 us of exposed latency; now 6 us.
__global__ void __launch_bounds__(256)
    k_mlp_reduce_adam(const float *__restrict__ part, int nparts, float *__restrict__ grad_out,
                      float *__restrict__ loss_out, float *__restrict__ params, float *__restrict__ m1,
                      float *__restrict__ m2, uint16_t *__restrict__ wb, float lr, float beta1, float beta2, float eps,
                      float c1, float c2, int adam) {
    __shared__ float s_g[8][32];
    const int lane = threadIdx.x & 31, group = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane;
    float g = 0.f;
    if (p <= kMlpParams) {
#pragma unroll 8
        for (int c = group; c < nparts; c += 8) g += part[(size_t)c * (kMlpParams + 1) + p];
    }
    s_g[group][lane] = g;
    __syncthreads();
    if (group != 0 || p > kMlpParams) return;
#pragma unroll
    for (int h = 1; h < 8; h++) g += s_g[h][lane];
    if (grad_out) grad_out[p] = g;
    if (p == kMlpParams) {
        if (loss_out) *loss_out = g;
        return;
    }
    if (!adam) return;
    const float a = beta1 * m1[p] + (1.f - beta1) * g;
    const float b = beta2 * m2[p] + (1.f - beta2) * g * g;
    m1[p] = a;
    m2[p] = b;
    const float w = params[p] - lr * (a * c1) / (sqrtf(b * c2) + eps);
    params[p] = w;
    store_wb(wb, p, w);
}

__global__ void k_mlp_refresh_wb(const float *__restrict__ params, uint16_t *__restrict__ wb) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kMlpParams) return;
    store_wb(wb, p, params[p]);
}

}  // namespace

// ---- host launchers ----------------------------------------------------------------------------
size_t mlp_fwd_smem() { return sizeof(FwdSmem); }
size_t mlp_train_smem() { return sizeof(TrainSmem); }

cudaError_t mlp_configure() {
    cudaError_t e = cudaFuncSetAttribute(k_mlp_predict, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FwdSmem));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_jc_warm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FwdSmem));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem));
}

void launch_mlp_predict(cudaStream_t s, const MlpDev &m, const float *x, int64_t n, float *y, uint32_t *status,
                        int grid) {
    k_mlp_predict<<<grid, kTile, sizeof(FwdSmem), s>>>(m, x, n, y, status);
}

void launch_mlp_predict_warp(cudaStream_t s, const MlpDev &m, const float *x, int64_t n, float *y, int grid) {
    k_mlp_predict_warp<<<grid, 256, 0, s>>>(m, x, n, y);
}

void launch_jc_warm(cudaStream_t s, int grid, const KConsts &K, const SortedFields32 &B, const FixedFields32 &F,
                    const ToolDev *tool, const MlpDev &m, int32_t *secant_iters, uint32_t *status) {
    k_jc_warm<<<grid, kTile, sizeof(FwdSmem), s>>>(K, B, F, tool, m, secant_iters, status);
}

void launch_mlp_grad(cudaStream_t s, int grid, const MlpDev &m, const float *x, const float *t, const int32_t *idx,
                     int64_t nb, float *part, uint32_t *status) {
    k_mlp_grad<<<grid, kTrainThreads, sizeof(TrainSmem), s>>>(m, x, t, idx, nb, 1.f / (float)nb, part, status);
}

void launch_mlp_reduce_adam(cudaStream_t s, const float *part, int nparts, float *grad_out, float *loss_out,
                            float *params, float *m1, float *m2, uint16_t *wb, float lr, float beta1, float beta2,
                            float eps, float c1, float c2, bool adam) {
    k_mlp_reduce_adam<<<div_up(kMlpParams + 1, 32), 256, 0, s>>>(part, nparts, grad_out, loss_out, params, m1, m2,
                                                                  wb, lr, beta1, beta2, eps, c1, c2, adam ? 1 : 0);
}

void launch_mlp_refresh_wb(cudaStream_t s, const float *params, uint16_t *wb) {
    k_mlp_refresh_wb<<<div_up(kMlpParams, 256), 256, 0, s>>>(params, wb);
}

}  // namespace sphfem
