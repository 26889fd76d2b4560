// interactions.cu -- neighbour sums of do_interactions_monaghan
// (interactions_gpu.cu:143-379: velocity gradient, stress divergence with
// Gray-Monaghan artificial stress, Monaghan artificial viscosity, XSPH and
// Brookshaw heat conduction) on sm_103a.
//
// One thread (FP32) or a few lanes (FP64) per particle in sorted order.
// Neighbours are visited column by column: the cells (ii, gj-R .. gj+R) of one grid
// column are consecutive keys, so their particles form one contiguous slot range [offsets[c0],
// offsets[c1+1]) -- the reference's visiting order (ii outer, jj inner,
// sorted order inside a cell) without per-cell bookkeeping.
//
// Out-of-support candidates are skipped: in the reference they run the full
// body with W = dW = 0 and add exact zeros (interactions_gpu.cu:230-337), so
// skipping them changes no sum.  Per-neighbour quotients that depend only on
// the neighbour ((S-p)/rho^2, mass/rho, sqrtf(K/rho)) come precomputed in the
// neighbour record; constant factors (mass, -eps*mass, 2*alpha) are applied
// once after the loop.  These reassociations change results by O(1e-16)
// relative.
//
// Fused mode adds, per particle, the rest of the particle chain up to the
// return mapping: do_material_stress_rate_jaumann, do_contmech_continuity /
// _momentum / _advection (actions_gpu.cu:280-314,626-687), correct
// (leap_frog.cu:71-96), do_material_fric_heat_gen_FEM_v21
// (actions_gpu.cu:345-420) and do_plasticity_johnson_cook
// (actions_gpu.cu:689-754).  Correct writes the start-of-step arrays in
// place (only this thread touches them); neighbours read the predicted state
// from the records, so there is no read/write race.
#include "interact64.cuh"

namespace sphfem {

// Launch shapes of the fused FP32K neighbour-sum kernel: (threads per block,
// minimum resident blocks per SM, staged records: 0 = global loads, lanes per
// particle).  Variant 0 is the default: 6 blocks (24 warps) per SM at 79
// registers (on grids of few waves without that bound, few_waves32).  On the
// 4.19 M lattice 128x6 and 256x3 are within 0.2 % of each other, 64x12, 64x8 and 128x4 1-2 % behind, 128x5 and 64x10 5 %; on the
// 12,000-particle cut the shapes with 2 and 4 lanes per particle are ahead.
const int kInteractVariants[][4] = {{128, 6, 0, 1},   {64, 12, 0, 1},   {64, 8, 0, 1},     {128, 4, 0, 1},
                                    {256, 3, 0, 1},   {256, 1, 0, 1},   {128, 3, 640, 1},  {128, 2, 1024, 1},
                                    {64, 6, 384, 1},  {256, 2, 1024, 1}, {128, 6, 0, 2},    {128, 6, 0, 4},
                                    {128, 5, 0, 1},   {64, 10, 0, 1}};

int interact_variant_count() { return (int)(sizeof(kInteractVariants) / sizeof(kInteractVariants[0])); }
void interact_variant_shape(int v, int *block, int *min_blocks, int *staged, int *lanes) {
    *block = kInteractVariants[v][0];
    *min_blocks = kInteractVariants[v][1];
    *staged = kInteractVariants[v][2];
    *lanes = kInteractVariants[v][3];
}

// SMs of the current device.
int sm_count() {
    static int sms[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int &n = sms[dev & 63];
    if (!n) {
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 152;
    }
    return n;
}

// Threads per block of the per-particle kernels with FP64 work: the largest of 256, 128,
// 64 that still gives every SM two blocks, else 32.  The FP64 pipe is narrow, so
// a small system (the reference's own cases are 7k-12k particles) must spread
// over all SMs rather than fill a few.  Results do not depend on it: these kernels'
// particles do not share their work.
int fp64_block(int N) {
    const int n = sm_count();
    for (int kb : {256, 128, 64})
        if (div_up(N, kb) >= 2 * n) return kb;
    return 32;
}

// ---- interactions_gpu.cu:84-140 do_interactions_heat_pse (FP64) --------------------------
// T_t = alpha * sum_j (T_j - T_i) W2(r_ij, h_i) m / rho_j over every particle of
// the 5x5 block of cells of edge h around the particle's cell (no support
// cut-off, blanked neighbours included), W2 = 4 / (h^4 pi) exp(-|r|^2 / h^2)
// (kernels.cuh:67-84).  Reads the predicted state from the FP64 records; the
// block's columns are contiguous slot ranges as in the neighbour sums.
// Bound by the FP64 pipe and, on the reference's own size, by the latency of its
// chains: the Gaussian and its product with the volume run on the integer pipes
// (6 FP64 operations a candidate instead of about 26) and kPseLanes lanes share a
// particle.  7,355 particles: 92 -> 14 us; 121,620: 471 -> 110 us; 490,072: 1.45 -> 0.42 ms.
constexpr int kPseLanes = 8;
// The term of a candidate whose numbers the mantissa form does not take.
static __device__ __noinline__ double pse_weight_general(double rr2, double inv_h2, double vol) {
    return exp(-rr2 * inv_h2) * vol;
}
__global__ void __launch_bounds__(128) k_heat_pse64(int N, KConsts K, const int32_t *__restrict__ offsets,
                                                    const dbl4 *__restrict__ rec,
                                                    const int32_t *__restrict__ hashes, double *__restrict__ T_t) {
    begin_after(offsets, rec, hashes, T_t);
    const int k = (int)(blockIdx.x * 128u + threadIdx.x) / kPseLanes, sub = (int)threadIdx.x % kPseLanes;
    const int kk = min(k, N - 1);
    const dbl4 i0 = ld_nc(rec + 4 * kk), i2 = ld_nc(rec + 4 * kk + 2), i3 = ld_nc(rec + 4 * kk + 3);
    const int fi = (int)__double_as_longlong(i3.w);
    const bool live = k < N && !(fi & kFlagBlanked);
    const double xi = i0.x, yi = i0.y, Ti = i3.z;
    const double h2 = i2.z * i2.z;
    const bool plain = !fix_range(h2);
    // log2(e) / h^2
    const Fix64 ch = fix_norm(Fix64{0xb8aa3b295c17f0bcull, -63} * fix_recip(plain ? 1. : h2));
    double sum = 0.;
    const int hash = hashes[kk];
    const sph_geom_constants &g = K.g;
    if (live && hash >= 0 && hash < g.num_cell) {
        const int gi = hash / g.ny, gj = hash - gi * g.ny;
        int ii = max(gi - 2, 0);
        const int ii1 = min(gi + 3, g.nx), lo_j = max(gj - 2, 0), hi_j = min(gj + 3, g.ny);
        int j = __ldg(offsets + ii * g.ny + lo_j) + sub, j1 = __ldg(offsets + ii * g.ny + hi_j);
        while (true) {   // every kPseLanes-th candidate of the columns' ranges, end to end
            while (j >= j1 && ++ii < ii1) {
                j += __ldg(offsets + ii * g.ny + lo_j) - j1;
                j1 = __ldg(offsets + ii * g.ny + hi_j);
            }
            if (j >= j1) break;
            const dbl4 n0 = ld_nc(rec + 4 * j), n3 = ld_nc(rec + 4 * j + 3);
            const double ex = n0.x - xi, ey = n0.y - yi;
            const double rr2 = ex * ex + ey * ey;
            double w;
            const Fix64 y = fix_norm(fix_of(rr2) * ch);
            if (plain || !fix_range(n3.y) || (uint32_t)__double2hiint(rr2) >= 0x7ff00000u) {
                w = pse_weight_general(rr2, 1. / h2, n3.y);
            } else {
                w = y.e + 63 > 10 ? 0. : fix_double(fix_exp2(y, true) * fix_of(n3.y));
            }
            sum += (n3.z - Ti) * w;
            j += kPseLanes;
        }
    }
    __syncwarp();
#pragma unroll
    for (int o = 1; o < kPseLanes; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (!live || sub != 0) return;
    // the reference binds the tool flags (doubles) for N ints, half the array
    // (interactions_gpu.cu:448): from index N/2 on its fetch reads zero
    const double alpha = ((fi & kFlagTool) && k < N / 2) ? K.c.trml_tool_sph.alpha : K.c.trml_wp.alpha;
    T_t[k] = alpha * (fix_div(4., h2 * h2 * kRigidPi) * sum);
}

// FP32-compensated form of the PSE sum over the FP32 records: positions as
// offsets from the cell corners (cells of edge h), the Gaussian with expf, the
// sum Kahan-compensated; T_t written in FP64.
template <class TT>   // T_t: double (staged call, FP64 arrays) or float (the compact state)
__global__ void __launch_bounds__(kBlock) k_heat_pse32(int N, KConsts K, const int32_t *__restrict__ offsets,
                                                       const float4 *__restrict__ rec,
                                                       const int32_t *__restrict__ hashes, TT *__restrict__ T_t) {
    begin_after(offsets, rec, hashes, T_t);
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= N) return;
    const float4 *rec_c = rec + 2 * (size_t)N, *rec_d = rec + 3 * (size_t)N;   // the records' last two quarters
    const float4 i0 = rec[k];
    const int fi = __float_as_int(i0.z);
    if (fi & kFlagBlanked) return;
    const float xri = i0.x, yri = i0.y, hi = i0.w, Ti = rec_d[k].w;
    const double alpha = ((fi & kFlagTool) && k < N / 2) ? K.c.trml_tool_sph.alpha : K.c.trml_wp.alpha;
    const float h2 = hi * hi;
    const float c = 4.f / (h2 * h2 * (float)kRigidPi);
    const float inv_h2 = 1.f / h2;
    const float cell = K.f.cell;
    KahanF sum = {};
    const int hash = hashes[k];
    const sph_geom_constants &g = K.g;
    if (hash >= 0 && hash < g.num_cell) {
        const int gi = hash / g.ny, gj = hash - gi * g.ny;
        const int lo_i = max(gi - 2, 0), hi_i = min(gi + 3, g.nx);
        const int lo_j = max(gj - 2, 0), hi_j = min(gj + 3, g.ny);
        for (int ii = lo_i; ii < hi_i; ii++) {
            const float dxc = (float)(gi - ii) * cell;
            const int j1 = __ldg(offsets + ii * g.ny + hi_j);
#pragma unroll 4   // several neighbours' loads in flight (the kernel waits on loads, not on math)
            for (int j = __ldg(offsets + ii * g.ny + lo_j); j < j1; j++) {
                const float4 n0 = rec[j];
                const float dx = dxc + (xri - n0.x);
                const float dy = (float)(gj - (__float_as_int(n0.z) & kRowMask)) * cell + (yri - n0.y);
                const float w2 = c * expf(-(dx * dx + dy * dy) * inv_h2);
                sum.add((rec_d[j].w - Ti) * w2 * rec_c[j].w);
            }
        }
    }
    T_t[k] = alpha * (double)sum.s;
}

void launch_heat_pse(cudaStream_t s, int N, const KConsts &K, const int32_t *offsets, const StepScratch &W,
                     const SortedFields32 &B) {
    const int tb = fp64_block(N);
    launch_after(s, k_heat_pse32<float>, div_up(N, tb), tb, 0, N, K, offsets, W.rec32, B.hash, B.T_t);
}

void launch_heat_pse(cudaStream_t s, int N, const KConsts &K, const int32_t *offsets, const StepScratch &W,
                     const SortedFields &B) {
    if (K.precision == SPH_PREC_FP32K) {
        const int tb = fp64_block(N);
        k_heat_pse32<<<div_up(N, tb), tb, 0, s>>>(N, K, offsets, W.rec32, B.hash, B.T_t);
        return;
    }
    launch_after(s, k_heat_pse64, div_up((int64_t)N * kPseLanes, 128), 128, 0, N, K, offsets, W.rec64, B.hash, B.T_t);
}

void launch_interactions32_fused(cudaStream_t s, int N, const KConsts &K, const int32_t *offsets,
                                 const SortedFields32 &B, const FixedFields32 &F, const StepScratch &W,
                                 const SegDev &seg, const ToolDev *tool, int variant) {
    launch_i32_variant<false>(s, N, K, offsets, B, F, W, seg, tool, variant, MlpDev{});
}

void launch_interactions(cudaStream_t s, int N, const KConsts &K, const int32_t *offsets, const SortedFields &B,
                         const FixedFields &F, const StepScratch &W, const SegDev &seg, const ToolDev *tool,
                         bool fused, int variant) {
    const int grid = div_up(N, kBlock);
    if (K.precision == SPH_PREC_FP32K) {
        // the fused FP32K step runs on the compact state (launch_interactions32_fused)
        k_interact32<false><<<grid, kBlock, 0, s>>>(N, K, offsets, W.rec32, W.cand32, B, F, seg, tool, W.secant_iters,
                                                    W.status, 0, MlpDev{});
    } else {
        const int g64 = div_up(N, kParts64);
        if (fused)
            launch_after(s,
                         three_blocks(N)   ? k_interact64<kMapQuads, 3>
                         : map_by_quads(N) ? k_interact64<kMapQuads>
                                           : k_interact64<kMapLane>,
                         g64, kThreads64, 0, N, K, offsets, W.rec64, W.cand32, B, F, seg, tool,
                         W.secant_iters, W.status);
        else
            k_interact64<kMapNone><<<g64, kThreads64, 0, s>>>(N, K, offsets, W.rec64, W.cand32, B, F, seg, tool,
                                                           W.secant_iters, W.status);
    }
}

}  // namespace sphfem
