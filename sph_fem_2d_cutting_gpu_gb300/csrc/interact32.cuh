// interact32.cuh -- the FP32 neighbour-sum kernel with Kahan-compensated
// sums (k_interact32), its fused epilogue and launch shapes; included by
// interactions.cu (the plain fused step and the staged call) and
// interactions_mlp.cu (the fused step with the learned warm start folded into
// its epilogue).  The sums are described in interactions.cu's header.
//
// Bound: instruction issue (74 % busy) and the L1's passes (56 % of peak), with 24
// warps per SM.  The candidate entries are read four to a load and tested without
// decoding (cand_pack32), every candidate is stored and the list grows past the ones
// that are in, the spline and the viscosity are selections instead of branches, sums
// and vectors use the packed FP32 instructions, and a record's quarters lie in four
// arrays (put_rec32): 9,100 instructions a warp instead of 10,440 and 1,940 L1 passes
// instead of 2,640.  Every pair term is formed in the order that it was in before,
// so the results are the same bit for bit.  4,194,304-particle lattice (2h cells) 1.453 ->
// 1.249 ms, 640,000-particle cut 257 -> 217 us, 12 cuts of 1.33 M particles 511 -> 427 us,
// 121,620-particle rigid cut (cells of h) 63 -> 50 us, 12,000-particle cut 39 -> 32 us.
// Products with a common factor as scalars instead of packed with the factor doubled,
// two pairs a turn, or the list entry fetched a turn ahead were 0-2 % slower.
#pragma once

#include <type_traits>

#include "async.cuh"
#include "launch.cuh"
#include "mlp_warp.cuh"
#include "rigid.cuh"

namespace sphfem {

// Kahan-compensated FP32 accumulator.
struct KahanF {
    float s, c;
    __device__ __forceinline__ void add(float v) {
        float y = v - c;
        float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    // Adds the partner lane's (s, c) (lane ^ o within mask): the two sums by an
    // error-free two-sum, whose rounding error joins the compensations.
    __device__ __forceinline__ void merge(unsigned mask, int o) {
        const float so = __shfl_xor_sync(mask, s, o), co = __shfl_xor_sync(mask, c, o);
        const float t = s + so;
        const float bp = t - s;
        const float e = (s - (t - bp)) + (so - bp);
        c = (c + co) - e;
        s = t;
    }
};

// Two FP32 values in a register pair, and the packed instructions on them (each half
// rounded as by the scalar one): half the issue slots, which bound this kernel.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pk(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ F2 pk(float a) { return pk(a, a); }
__device__ __forceinline__ float f2lo(F2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return x;
}
__device__ __forceinline__ float f2hi(F2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return y;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

// Two KahanF accumulators side by side; n holds the negated compensations.
struct Kahan2 {
    F2 s, n;
    // adds a * b (the products enter the compensated sums unrounded)
    __device__ __forceinline__ void add_product(F2 a, F2 b) { fold(fma2(a, b, n)); }
    __device__ __forceinline__ void add(F2 v) { fold(v + n); }
    __device__ __forceinline__ void fold(F2 y) {
        const F2 t = s + y;
        n = y - (t - s);
        s = t;
    }
    __device__ __forceinline__ KahanF first() const { return {f2lo(s), -f2lo(n)}; }
    __device__ __forceinline__ KahanF second() const { return {f2hi(s), -f2hi(n)}; }
};

// Hardware approximations of positive normal arguments, without the library
// functions' scaling of subnormal ones.
__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Four candidate entries of an aligned group.
__device__ __forceinline__ void ld_cand4(const float2 *p, float2 (&c)[4]) {
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(c[0].x), "=f"(c[0].y), "=f"(c[1].x), "=f"(c[1].y), "=f"(c[2].x), "=f"(c[2].y), "=f"(c[3].x),
                   "=f"(c[3].y)
                 : "l"(p));
}

// The row difference gj - row of an FP64 candidate entry (cand_pack64): its y carries the
// row modulo 8 in the three lowest bits, and |gj - row| <= kMaxStencil = 3, so the
// low three bits of the difference, sign-extended, are the difference.
__device__ __forceinline__ int cand_row_diff(int gj, float cy) {
    return (int)(((unsigned)gj - (unsigned)__float_as_int(cy)) << 29) >> 29;
}

// In-support neighbours collected per pass of the pair loops.  With h = 1.7 dx
// a particle has about 36 (a disc of radius 2h): 40 covers nearly all of them
// in one pass.  A second, short pass costs more than its share: the lanes of a
// warp hold 0 to 10 pairs in it, and it re-enters the candidate scan (36 or 32
// entries: 13-15 % slower on the 4.19 M lattice).  Larger lists take shared
// memory from the L1 that serves the neighbour records: at 128 threads x 6
// blocks, 40 entries take 120 KB of shared memory per SM, 48 take 144 KB and
// were 1.3 % slower (44: the same as 48).
constexpr int kChunk32 = 40;

// Sums of the fused FP32 pair loop, each Kahan-compensated.  The epilogue needs
// the stress divergence and the artificial viscosity only through the
// acceleration (actions_gpu.cu:641-671: vel_t = visc + (S_der.x + S_der.y) +
// forces / m), so both go into one sum per component: nine sums instead of
// the staged form's thirteen.
struct Acc32Fused {
    Kahan2 vd01, vd23, a, xt;
    KahanF tl;
};

// A particle blanked before the step skips the neighbour sums, the corrector and
// the return mapping, but the rigid tool's do_material_fric_heat_gen
// (actions_gpu.cu:316-343) has no blanked test and still heats it.
template <class SF>
__device__ __forceinline__ void rigid_heat_blanked(int k, const KConsts &K, const SF &B) {
    if (!K.rigid || K.c.trml_wp.eta == 0. || flag_nonzero(B.tool_particle[k])) return;
    const double T0 = B.T[k];
    double T = T0;
    rigid_fric_heat_one(K, K.dt, K.rigid->vel, d2(B.vel[k]), d2(B.ft[k]), d2(B.n[k]), T);
    if (T != T0) put(B.T[k], T);
}

// FP32-compensated epilogue on the compact FP32 state: the rates (Jaumann,
// continuity, momentum, advection) and the return mapping in FP32; the
// corrector keeps positions and density in FP64.  vd, sd, vt, xt as in the
// FP64 epilogue.
// kMlp: a yielding particle only sets `pending`; its return mapping runs after
// the warp's forward passes of the learned warm start (jc_warm_warp).
template <bool kMlp>
__device__ __forceinline__ void fused_epilogue32(int k, const KConsts &K, const SortedFields32 &B,
                                                 const FixedFields32 &F, const SegDev &seg,
                                                 const ToolDev *__restrict__ tool, int32_t *__restrict__ secant_iters,
                                                 uint32_t *status, bool is_tool, float2 vel_pred, float rho_pred,
                                                 float4 vd, float4 sd, float2 vt, float2 xt, bool thermal, float T_t_new,
                                                 bool &pending) {
    const ToolDev &tc = tool[case_of_hash(K, B.hash[k])];   // the particle's case (time step, tool)
    const double dt = tc.dt;
    const float dtf = tc.dtf, hdtf = tc.hdtf;
    const float inv_mass = K.f.inv_mass;
    const float4 S0 = B.S[k];
    float4 St;
    float2 pos_t, vel_t;
    float rho_t;
    if (!is_tool) {
        const float4 Sto = B.S_t[k];
        float4 Sp = make_float4(fmaf(hdtf, Sto.x, S0.x), fmaf(hdtf, Sto.y, S0.y), fmaf(hdtf, Sto.z, S0.z),
                                fmaf(hdtf, Sto.w, S0.w));
        St = jaumann_f32(K.f.G, vd, Sp);
        rho_t = -rho_pred * (vd.x + vd.w);
        const float2 fc = B.fc[k], ft = B.ft[k];
        vel_t.x = vt.x + ((sd.x + sd.y) + (fc.x + ft.x) * inv_mass);
        vel_t.y = vt.y + ((sd.z + sd.w) + (fc.y + ft.y) * inv_mass);
        pos_t.x = xt.x + vel_pred.x;
        pos_t.y = xt.y + vel_pred.y;
        B.S_t[k] = St;
        B.rho_t[k] = rho_t;
    } else {
        St = B.S_t[k];
        rho_t = B.rho_t[k];
        if (K.thermal_pse) {   // PSE build: tool particles leave the sums unwritten
            vel_t = B.vel_t[k];
            pos_t = B.pos_t[k];
        } else {
            vel_t = vt;
            pos_t = xt;
        }
    }
    const float T_t = thermal ? T_t_new : B.T_t[k];
    B.pos_t[k] = pos_t;
    B.vel_t[k] = vel_t;
    if (thermal) B.T_t[k] = T_t;
    // corrector (leap_frog.cu:71-96)
    double2 pos = B.pos[k];
    pos.x = pos.x + dt * (double)pos_t.x;
    pos.y = pos.y + dt * (double)pos_t.y;
    B.pos[k] = pos;
    const float2 v0 = B.vel[k];
    const float2 vel = make_float2(fmaf(dtf, vel_t.x, v0.x), fmaf(dtf, vel_t.y, v0.y));
    B.vel[k] = vel;
    float4 S = make_float4(fmaf(dtf, St.x, S0.x), fmaf(dtf, St.y, S0.y), fmaf(dtf, St.z, S0.z), fmaf(dtf, St.w, S0.w));
    const double rho = B.rho[k] + dt * (double)rho_t;
    B.rho[k] = rho;
    float T = fmaf(dtf, T_t, B.T[k]);
    uint32_t st = 0;
    bool blanked = false;
    if (K.has_tool) {   // friction heat (actions_gpu.cu:345-420) for particles in contact
        const int on = B.on_seg[k];
        if (on >= 0 && on < seg.n) {
            double Td = (double)T, bl = 0.;
            st |= fric_heat_one(K, dt, tc.vel, make_double2(vel.x, vel.y), d2(B.ft[k]), d2(B.n[k]), d2(B.fc[k]), rho,
                                (double)B.eps_pl[k], on, seg.n, Td, bl, seg.fric_heat, seg.wear);
            T = (float)Td;
            blanked = flag_is_one(bl);
        }
    } else if (K.rigid && !is_tool && K.c.trml_wp.eta != 0.) {   // actions_gpu.cu:316-343
        double Td = (double)T;
        rigid_fric_heat_one(K, dt, K.rigid->vel, make_double2(vel.x, vel.y), d2(B.ft[k]), d2(B.n[k]), Td);
        T = (float)Td;
    }
    if (K.c.plastic && !is_tool && !blanked) {   // return mapping (actions_gpu.cu:689-754)
        const JcF32 &j = K.f.jc;
        float eps_pl = B.eps_pl[k], eps_pl_dot = B.eps_pl_dot[k];
        int it = 0;
        if constexpr (kMlp) {
            JcTrial tr;
            if (jc_trial_f32(j, S, F.p[k], eps_pl, eps_pl_dot, T, tr)) pending = true;
            else B.eps_pl_dot[k] = 0.f;
        } else if (K.jc_list) {
            // learned warm start: the trial state is stored below and a yielding
            // particle finishes its return mapping in k_jc_warm
            JcTrial tr;
            if (jc_trial_f32(j, S, F.p[k], eps_pl, eps_pl_dot, T, tr)) {
                const unsigned mask = __activemask();
                const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
                int base = 0;
                if (lane == leader) base = atomicAdd(K.jc_list_count, __popc(mask));
                base = __shfl_sync(mask, base, leader);
                K.jc_list[base + __popc(mask & ((1u << lane) - 1u))] = k;
            } else {
                B.eps_pl_dot[k] = 0.f;
            }
        } else {
            st |= plasticity_f32(K, j, dtf, tc.inv_dtf, S, F.p[k], (float)rho, eps_pl, eps_pl_dot, T, blanked, &it);
            B.eps_pl[k] = eps_pl;
            B.eps_pl_dot[k] = eps_pl_dot;
        }
        if (secant_iters) secant_iters[k] = it;
    }
    B.S[k] = S;
    B.T[k] = T;
    if (blanked) B.blanked[k] = 1.f;
    if (st) set_status(status, st);
}

// ---- FP32 with Kahan-compensated sums --------------------------------------------------
// Staged blocks: the records of the block's cells and their stencil halo,
// one contiguous run per grid column (cells are column-major in the sorted
// order), copied into shared memory by the bulk-copy engine before the pair
// loops.  Staged only when all of the block's particles lie in one grid column
// and the region holds at most `cap` records; otherwise global loads.
struct StageHdr {
    int staged, ix, r_lo, r_hi, c_lo;
    int delta[2 * kMaxStencil + 1];   // shared slot minus global record index, per column
};

template <class SF>
__device__ __forceinline__ void stage_issue(int vb, int N, int kB, const KConsts &K, const int32_t *__restrict__ offsets,
                                            const float4 *__restrict__ rec, const SF &B, int cap,
                                            float4 *srec, StageHdr &h, uint32_t mbar) {
    const sph_geom_constants &g = K.g;
    const int R = g.stencil;
    const int b0 = vb * kB;
    const int hf = B.hash[b0], hl = B.hash[min(b0 + kB, N) - 1];
    h.staged = 0;
    if (hf < 0 || hl >= g.num_cell || hl < hf) return;
    const int ix = hf / g.ny;
    if (hl / g.ny != ix) return;
    const int r_lo = max(hf - ix * g.ny - R, 0), r_hi = min(hl - ix * g.ny + R, g.ny - 1);
    const int c_lo = max(ix - R, 0), c_hi = min(ix + R, g.nx - 1);
    int total = 0, start[2 * kMaxStencil + 1], len[2 * kMaxStencil + 1];
    for (int c = c_lo; c <= c_hi; c++) {
        start[c - c_lo] = __ldg(offsets + c * g.ny + r_lo);
        len[c - c_lo] = __ldg(offsets + c * g.ny + r_hi + 1) - start[c - c_lo];
        h.delta[c - c_lo] = total - start[c - c_lo];
        total += len[c - c_lo];
    }
    if (total <= 0 || total > cap) return;
    mbar_init(mbar);
    mbar_arrive_expect_tx(mbar, (uint32_t)total * 64u);
    const bool issue = !(K.test_faults & SPH_TEST_SKIP_BULK_COPY);   // a test lets the wait run out
    for (int c = c_lo; c <= c_hi; c++)
        if (issue && len[c - c_lo] > 0)
            for (int q = 0; q < 4; q++)
                bulk_g2s(smem_u32(srec + q * cap + start[c - c_lo] + h.delta[c - c_lo]),
                         rec + (size_t)q * N + start[c - c_lo], (uint32_t)len[c - c_lo] * 16u, mbar);
    h.staged = 1;
    h.ix = ix;
    h.r_lo = r_lo;
    h.r_hi = r_hi;
    h.c_lo = c_lo;
}

// L2 prefetch by one thread at block start, overlapped with the neighbour loops:
// the block's slice of the start-of-step state its epilogue reads, and, when
// the block lies in one grid column, the neighbour records of its stencil
// (one contiguous run of rows per column).  Hints only: every range lies
// inside its array.
template <class SF, class FF>
__device__ __forceinline__ void block_prefetch_l2(int vb, int N, int kB, const KConsts &K,
                                                  const int32_t *__restrict__ offsets, const float4 *__restrict__ rec,
                                                  const float2 *__restrict__ cand, const SF &B, const FF &F) {
    const int b0 = vb * kB;
    const uint32_t n = (uint32_t)min(kB, N - b0);
    prefetch_l2_bulk(B.S + b0, n * (uint32_t)sizeof(B.S[0]));
    prefetch_l2_bulk(B.S_t + b0, n * (uint32_t)sizeof(B.S_t[0]));
    prefetch_l2_bulk(B.pos + b0, n * 16u);
    prefetch_l2_bulk(B.vel + b0, n * (uint32_t)sizeof(B.vel[0]));
    prefetch_l2_bulk(B.fc + b0, n * (uint32_t)sizeof(B.fc[0]));
    prefetch_l2_bulk(B.ft + b0, n * (uint32_t)sizeof(B.ft[0]));
    prefetch_l2_bulk(B.rho + b0, n * 8u);
    prefetch_l2_bulk(B.T + b0, n * (uint32_t)sizeof(B.T[0]));
    prefetch_l2_bulk(B.eps_pl + b0, n * (uint32_t)sizeof(B.eps_pl[0]));
    prefetch_l2_bulk(B.eps_pl_dot + b0, n * (uint32_t)sizeof(B.eps_pl_dot[0]));
    prefetch_l2_bulk(F.p + b0, n * (uint32_t)sizeof(F.p[0]));
    const sph_geom_constants &g = K.g;
    const int R = g.stencil;
    const int hf = B.hash[b0], hl = B.hash[b0 + (int)n - 1];
    if (hf < 0 || hl >= g.num_cell || hl < hf) return;
    const int ix = hf / g.ny;
    if (hl / g.ny != ix) return;
    const int r_lo = max(hf - ix * g.ny - R, 0), r_hi = min(hl - ix * g.ny + R, g.ny - 1);
    for (int c = max(ix - R, 0); c <= min(ix + R, g.nx - 1); c++) {
        const int s0 = __ldg(offsets + c * g.ny + r_lo), s1 = __ldg(offsets + c * g.ny + r_hi + 1);
        if (s1 > s0) {
            for (int q = 0; q < 4; q++) prefetch_l2_bulk(rec + (size_t)q * N + s0, (uint32_t)(s1 - s0) * 16u);
            const int a0 = s0 & ~1;   // 16-byte aligned start; the size is rounded down
            prefetch_l2_bulk(cand + a0, (uint32_t)(s1 - a0) * 8u);
        }
    }
}

// kB threads per block, at least kMinB resident blocks per SM (a register
// budget for the compiler): the launch shapes the autotuner chooses from.
// kStaged: neighbour records from shared memory (dynamic: cap records + the
// pair lists).
// The fused form works on the compact FP32 state (SortedFields32 / FixedFields32);
// the staged form (sph_interactions_monaghan) on the FP64 arrays.
template <bool kFused>
using Sorted32Of = std::conditional_t<kFused, SortedFields32, SortedFields>;
template <bool kFused>
using Fixed32Of = std::conditional_t<kFused, FixedFields32, FixedFields>;

// kMlp (fused only): the learned warm start of the return mapping in the
// epilogue, one warp-wide forward pass per yielding particle; every lane of a
// warp reaches it, so the per-particle body returns from a lambda.
// One block of kB / kSplit particles, vb-th in sorted order (the kernel's
// blockIdx.x, or a persistent kernel's virtual block).  kSplit > 1 (small
// systems, fused form): kSplit consecutive lanes share a particle, each
// scanning every kSplit-th candidate of each stencil column; their sums are
// merged (compensated) before the epilogue, which the first lane runs.
template <bool kFused, int kB, bool kStaged, bool kMlp, int kSplit = 1>
__device__ __forceinline__ void interact32_block(int vb, int N, const KConsts &K, const int32_t *__restrict__ offsets,
                                                 const float4 *__restrict__ rec, const float2 *__restrict__ cand,
                                                 const Sorted32Of<kFused> &B,
                                                 const Fixed32Of<kFused> &F, const SegDev &seg,
                                                 const ToolDev *__restrict__ tool, int32_t *__restrict__ secant_iters,
                                                 uint32_t *status, int cap, const MlpDev &mlp) {
    static_assert(kFused || !kMlp, "the warm start is folded into the fused epilogue only");
    static_assert(kSplit == 1 || (kFused && !kStaged && 32 % kSplit == 0), "split lanes: fused, unstaged");
    constexpr int kPPB = kB / kSplit;   // particles per block
    const int k = vb * kPPB + (int)threadIdx.x / kSplit;
    const int sub = (int)threadIdx.x % kSplit;
    const unsigned gmask = ((1u << kSplit) - 1u) << ((threadIdx.x & 31u) & ~(unsigned)(kSplit - 1));
    if (kFused && threadIdx.x == 0) block_prefetch_l2(vb, N, kPPB, K, offsets, rec, cand, B, F);
    int (*s_list)[kB];
    const float4 *rec_b = rec + 2 * (size_t)N;   // the records' third and fourth quarters
    const float4 *nrec = rec;   // staged: the copies in shared memory, quarter by quarter
    __shared__ StageHdr s_hdr;
    __shared__ alignas(8) unsigned long long s_mbar;
    bool staged = false;
    if constexpr (kStaged) {
        extern __shared__ __align__(128) float4 s_dyn[];
        s_list = (int (*)[kB])(s_dyn + 4 * cap);
        if (threadIdx.x == 0) stage_issue(vb, N, kB, K, offsets, rec, B, cap, s_dyn, s_hdr, smem_u32(&s_mbar));
        __syncthreads();
        if (s_hdr.staged) {
            staged = mbar_wait(smem_u32(&s_mbar), 0);
            if (staged) {
                nrec = s_dyn;
            } else {   // copies late: report, wait once more (bounded) for them, use global loads
                if (threadIdx.x == 0) set_status(status, SPH_STATUS_COPY_TIMEOUT);
                mbar_wait(smem_u32(&s_mbar), 0);
            }
        }
    } else {
        __shared__ int s_list_st[kChunk32 + 1][kB];
        s_list = s_list_st;
    }
    bool pending = false;   // kMlp: this particle yields and waits for its warm start
    auto particle = [&]() {
    if (k >= N) return;
    const float4 i0 = rec[k];
    const int fi = __float_as_int(i0.z);
    if (fi & kFlagBlanked) {
        if (kFused && sub == 0) rigid_heat_blanked(k, K, B);   // one lane per particle
        return;
    }
    const bool tool_i = (fi & kFlagTool) != 0;
    const float4 i1 = rec[N + k], i2 = rec_b[k], i3 = rec_b[N + k];
    const float xri = i0.x, yri = i0.y, hi = i0.w;
    const float vix = i1.x, viy = i1.y, rhoi = i1.z, ci = i1.w;
    const float sAi = i2.x, sCi = i2.y, sBi = i2.z;
    const float Rxxi = i3.x, Ryyi = i3.y, Rxyi = i3.z, Ti = i3.w;
    const float thermal_alpha = (!tool_i) ? K.f.alpha_wp : K.f.alpha_tool_sph;
    const bool thermal = thermal_alpha != 0.f && !K.thermal_pse;   // Brookshaw build only
    const bool pse_tool = K.thermal_pse && tool_i;                  // PSE build: tool particles return at once
    const float h1 = 1.f / hi;
    const float fourh2 = 4.f * hi * hi;
    const float fac = (float)kPiFac * h1 * h1;
    const float alpha = K.f.alpha, beta = K.f.beta, eta2 = K.f.eta2;
    const float inv_wdp = K.f.inv_wdp;
    const float cell = K.f.cell;

    KahanF vd0 = {}, vd1 = {}, vd2 = {}, vd3 = {}, sd0 = {}, sd1 = {}, sd2 = {}, sd3 = {};
    KahanF vt0 = {}, vt1 = {}, xt0 = {}, xt1 = {}, tl = {};
    Acc32Fused af = {};
    // cubic spline (kernels.cuh:25-65) with the per-particle factors folded:
    // q > 1: W = fac/4 (2-q)^6, dW/(r dr) = -3/4 fac h1 (2-q)^2 / r;
    // q <= 1: W = fac (1 - 3/2 q^2 + 3/4 q^3), dW/(r dr) = fac h1^2 (-3 + 9/4 q)
    const float kwa = 0.25f * fac, kda = -0.75f * fac * h1;
    const float kwc = -1.5f * fac, kwd = 0.75f * fac;
    const float kde = -3.f * fac * h1 * h1, kdf = 2.25f * fac * h1 * h1;
    const int hash = B.hash[k];
    const sph_geom_constants &g = K.g;
    int gi = 0, gj = 0, ii = 0, hi_i = 0, lo_j = 0, hi_j = 0;
    int j = 0, j0 = 0, j1 = 0;   // the column's range [j0, j1); j: the next group of four, aligned
    const int R = g.stencil;
    bool done = true;
    if (hash >= 0 && hash < g.num_cell && !pse_tool) {
        gi = hash / g.ny;
        gj = hash - gi * g.ny;
        ii = max(gi - R, 0);
        hi_i = min(gi + R + 1, g.nx);
        lo_j = max(gj - R, 0);
        hi_j = min(gj + R + 1, g.ny);
        done = false;
    }
    // a particle whose stencil lies inside the staged region reads its neighbours'
    // records from shared memory (slot = global index + per-column delta); any other
    // uses global loads
    bool use_s = false;
    if constexpr (kStaged)
        use_s = staged && !done && gi == s_hdr.ix && lo_j >= s_hdr.r_lo && hi_j - 1 <= s_hdr.r_hi;
    // Pass 0 sums over the in-support neighbours.  In the reference every active
    // particle of the stencil (this one included) runs the pair body, with zero
    // kernel weights outside the support: exact zeros for finite data, but NaN
    // when one of the factors is NaN or infinite.  So a particle whose stencil
    // holds a record marked non-finite repeats its sums over every active
    // candidate with the reference's zero weights (pass 1).
    int marks = 0;   // OR of the flags of the candidates that the entries could not decide
    const float cell8 = 8.f * cell;
    const F2 cell_2 = pk(cell), x_i = pk(xri, yri), v_i = pk(vix, viy), s_i = pk(sAi, sCi), R_i = pk(Rxxi, Ryyi);
    const float rhoi_half = 0.5f * rhoi, hi_half = 0.5f * hi, ci_half = 0.5f * ci;
    // this particle in the entries' frame; one whose own entry could not decide takes all
    const bool take_all = (fi & (kFlagNonFinite | kFlagFar)) != 0;
    const float y8 = take_all ? __int_as_float(0x7fffffff) : cand_y8(yri, gj & 7, cell);
    const int undecided = kFlagNonFinite | kFlagFar;
    auto column = [&]() {   // the range of column ii
        j0 = __ldg(offsets + ii * g.ny + lo_j);
        j1 = __ldg(offsets + ii * g.ny + hi_j);
        j = (j0 & ~3) + 4 * sub;
    };
    auto sweep = [&](auto all_tag) {
    constexpr bool all = decltype(all_tag)::value;
    if (!done) column();
    while (!done) {
        // phase 1: collect the next in-support neighbours (column offset packed in 3 bits)
        // from the 8-byte candidate entries, four in one aligned load.  Every candidate is
        // stored, and the list grows past it if it is in.
        int *lp = &s_list[0][threadIdx.x];
        const int *const list = lp;
        while (lp <= list + (kChunk32 - 4) * kB) {
            if (j < j1) {
                const float xc = fmaf((float)(gi - ii), cell, xri);
                const int e = (j << 3) | (gi - ii + R), u0 = j - j0;
                const unsigned len = (unsigned)(j1 - j0);
                float2 c[4];
                ld_cand4(cand + j, c);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const float dx = xc - c[u].x, dd = y8 - c[u].y;
                    const float dy = fminf(fabsf(dd), cell8 - fabsf(dd));
                    const float rr2 = dx * dx + dy * dy;
                    *lp = e + 8 * u;
                    // NaN passes both tests of the distance
                    const bool in = ((unsigned)(u0 + u) < len) & (all | (!(rr2 >= fourh2) & !(rr2 < 1e-8f)));
                    lp += in ? kB : 0;
                }
                j += 4 * kSplit;
            } else {
                if (++ii >= hi_i) {
                    done = true;
                    break;
                }
                column();
            }
        }
        // phase 2: the pair body over the collected list, lanes in step.  No
        // software prefetch of the next record: the 32 registers it holds cost
        // more resident warps than it hides latency.
        for (const int *q0 = list; q0 < lp; q0 += kB) {
            const int e = *q0;
            const int jn = e >> 3;
            float4 n0, n1, n2, n3;   // the neighbour's 64-byte record
            if (use_s) {
                const float4 *r = nrec + (jn + s_hdr.delta[gi + R - (e & 7) - s_hdr.c_lo]);
                n0 = r[0];
                n1 = r[cap];
                n2 = r[2 * cap];
                n3 = r[3 * cap];
            } else {
                n0 = __ldg(rec + jn);
                n1 = __ldg(rec + N + jn);
                n2 = __ldg(rec_b + jn);
                n3 = __ldg(rec_b + N + jn);
            }
            const int fj = __float_as_int(n0.z);
            // the distance vector: cell offset times the cell edge, plus the offsets in the cells
            const F2 off = pk((float)((e & 7) - R), (float)(gj - (fj & kRowMask)));
            const F2 d = fma2(off, cell_2, x_i - pk(n0.x, n0.y));
            const float dx = f2lo(d), dy = f2hi(d);
            const float rr2 = dx * dx + dy * dy;
            // FP32 form: hardware reciprocal square root instead of sqrt and division; both
            // branches of the spline and a selection, so that the lanes stay together
            const float inv_r = rsqrt_approx(rr2);
            const float q = rr2 * inv_r * h1;
            const bool far = q > 1.f;
            // pass 1: cubic_spline's zero weights outside the support (kernels.cuh:37-39)
            bool zero_w = false, conduction_only = false;
            if (all || ((fj | fi) & (undecided | kFlagTool))) {   // rare
                const bool out = !(rr2 < fourh2 && rr2 >= 1e-8f);
                if (all) {
                    if (fj & kFlagBlanked) continue;
                    zero_w = out;
                } else if ((fj | fi) & undecided) {
                    marks |= fj | fi;
                    if (out || (fj & kFlagBlanked)) continue;
                }
                conduction_only = ((fj | fi) & kFlagTool) != 0;
            }
            if constexpr (kFused) {
                const float u = far ? 2.f - q : q, u2 = u * u;
                float w = far ? kwa * (u2 * u2 * u2) : fmaf(u2, fmaf(kwd, u, kwc), fac);
                float dwf = far ? kda * u2 * inv_r : fmaf(kdf, u, kde);
                if (all && zero_w) w = dwf = 0.f;
                if (thermal && (!all || !zero_w || rr2 > 1e-16f)) af.tl.add(n2.w * (Ti - n3.w) * dwf);
                if (conduction_only) continue;
                const F2 wg = pk(dwf) * d;   // grad W
                const F2 dv = pk(n1.x, n1.y) - v_i;
                const F2 tv = wg * pk(n2.w);
                af.vd01.add_product(pk(f2lo(dv)), tv);
                af.vd23.add_product(pk(f2hi(dv)), tv);
                float fab = w * inv_wdp;
                fab *= fab;
                fab *= fab;
                const F2 sd = fma2(pk(fab), R_i + pk(n3.x, n3.y), s_i + pk(n2.x, n2.y));
                const float sxy = fmaf(fab, Rxyi + n3.z, sBi + n2.z);
                const float vijposij = -(f2lo(dv) * dx + f2hi(dv) * dy);
                const float irho = rcp_approx(fmaf(0.5f, n1.z, rhoi_half));
                const float hij = fmaf(0.5f, n0.w, hi_half);
                const float muij = hij * vijposij * rcp_approx(fmaf(eta2 * hij, hij, rr2));
                const float pi = (-alpha * fmaf(0.5f, n1.w, ci_half) * muij + beta * muij * muij) * irho;
                const F2 sp = sd - pk(vijposij < 0.f ? pi : 0.f);   // viscosity of an approaching pair
                // acceleration / mass: (stress terms - viscosity) . grad W
                af.a.add(fma2(pk(f2lo(sp), sxy), pk(f2lo(wg)), pk(sxy, f2hi(sp)) * pk(f2hi(wg))));
                af.xt.add_product(pk(w * irho), dv);
            } else {
                float val, der;
                if (far) {
                    const float t = 2.f - q, t2 = t * t;
                    val = 0.25f * t2 * t2 * t2;
                    der = -0.75f * t2 * h1 * inv_r;
                } else {
                    val = 1.f - 1.5f * q * q * (1.f - 0.5f * q);
                    der = -3.0f * q * (1.f - 0.75f * q) * h1 * inv_r;
                }
                const float w = zero_w ? 0.f : val * fac;
                const float dwf = zero_w ? 0.f : der * fac;
                const float wx = dwf * dx, wy = dwf * dy;
                const float volj = n2.w;
                if (!conduction_only) {
                    const float dvx = n1.x - vix, dvy = n1.y - viy;
                    const float tx = wx * volj, ty = wy * volj;
                    vd0.add(dvx * tx);
                    vd1.add(dvx * ty);
                    vd2.add(dvy * tx);
                    vd3.add(dvy * ty);
                    float fab = w * inv_wdp;
                    fab *= fab;
                    fab *= fab;
                    const float ax = (sAi + n2.x) + fab * (Rxxi + n3.x);
                    const float ay = (sBi + n2.z) + fab * (Rxyi + n3.z);
                    const float az = (sCi + n2.y) + fab * (Ryyi + n3.y);
                    sd0.add(ax * wx);
                    sd1.add(ay * wy);
                    sd2.add(ay * wx);
                    sd3.add(az * wy);
                    const float vijposij = -(dvx * dx + dvy * dy);
                    const float irho = __fdividef(2.f, rhoi + n1.z);
                    if (vijposij < 0.f) {
                        const float cij = 0.5f * (ci + n1.w);
                        const float hij = 0.5f * (hi + n0.w);
                        const float muij = __fdividef(hij * vijposij, rr2 + eta2 * hij * hij);
                        const float piij = (-alpha * cij * muij + beta * muij * muij) * irho;
                        vt0.add(piij * wx);
                        vt1.add(piij * wy);
                    }
                    const float wr = w * irho;
                    xt0.add(wr * dvx);
                    xt1.add(wr * dvy);
                }
                if (thermal && (!zero_w || rr2 > 1e-16f)) tl.add(volj * (Ti - n3.w) * dwf);
            }
        }
    }
    };
    sweep(std::false_type{});
    if constexpr (kSplit > 1) {   // the particle's stencil as a whole
#pragma unroll
        for (int o = 1; o < kSplit; o <<= 1) marks |= __shfl_xor_sync(gmask, marks, o);
    }
    if (marks & kFlagNonFinite) {   // rare: the reference's full stencil with zero weights
        vd0 = vd1 = vd2 = vd3 = sd0 = sd1 = sd2 = sd3 = vt0 = vt1 = xt0 = xt1 = tl = KahanF{};
        af = Acc32Fused{};
        ii = max(gi - R, 0);
        done = false;
        sweep(std::true_type{});
    }
    if constexpr (kFused) {
        KahanF f[9] = {af.vd01.first(), af.vd01.second(), af.vd23.first(), af.vd23.second(), af.a.first(),
                       af.a.second(), af.xt.first(), af.xt.second(), af.tl};
        if constexpr (kSplit > 1) {   // merge the lanes' compensated sums; the first lane goes on
#pragma unroll
            for (int o = 1; o < kSplit; o <<= 1)
#pragma unroll
                for (int m = 0; m < 9; m++) f[m].merge(gmask, o);
            if (sub != 0) return;
        }
        const float mass = K.f.mass;
        const float xs = K.f.xs_mass;
        const float4 vd = make_float4(f[0].s, f[1].s, f[2].s, f[3].s);
        // the whole acceleration sum rides in sd.x / sd.z (vt zero): the epilogue adds sd.x + sd.y + vt.x
        const float4 sd = make_float4(mass * f[4].s, 0.f, mass * f[5].s, 0.f);
        const float2 xt = make_float2(xs * f[6].s, xs * f[7].s);
        const float T_t = thermal_alpha * (2.0f * f[8].s);
        // predicted velocity and density from this particle's record
        fused_epilogue32<kMlp>(k, K, B, F, seg, tool, secant_iters, status, tool_i, make_float2(vix, viy), rhoi, vd,
                               sd, make_float2(0.f, 0.f), xt, thermal, T_t, pending);
    } else {
        const float mass = K.f.mass;
        const float xs = K.f.xs_mass;
        const float4 vd = make_float4(vd0.s, vd1.s, vd2.s, vd3.s);
        const float4 sd = make_float4(mass * sd0.s, mass * sd1.s, mass * sd2.s, mass * sd3.s);
        const float2 vt = make_float2(-mass * vt0.s, -mass * vt1.s);
        const float2 xt = make_float2(xs * xt0.s, xs * xt1.s);
        const float T_t = thermal_alpha * (2.0f * tl.s);
        if (pse_tool) return;
        F.S_der[k] = mk4(sd.x, sd.y, sd.z, sd.w);
        F.v_der[k] = mk4(vd.x, vd.y, vd.z, vd.w);
        B.pos_t[k] = make_double2(xt.x, xt.y);
        B.vel_t[k] = make_double2(vt.x, vt.y);
        if (thermal) B.T_t[k] = (double)T_t;
    }
    };
    particle();
    if constexpr (kMlp) jc_warm_warp(K, B, F, tool, mlp, k, pending, secant_iters, status);
}

template <bool kFused, int kB = kBlock, int kMinB = 1, bool kStaged = false, bool kMlp = false, int kSplit = 1>
__global__ void __launch_bounds__(kB, kMinB) k_interact32(int N, KConsts K, const int32_t *__restrict__ offsets,
                                                       const float4 *__restrict__ rec,
                                                       const float2 *__restrict__ cand, Sorted32Of<kFused> B,
                                                       Fixed32Of<kFused> F, SegDev seg,
                                                       const ToolDev *__restrict__ tool,
                                                       int32_t *__restrict__ secant_iters, uint32_t *status,
                                                       int cap, MlpDev mlp) {
    begin_after(offsets, rec, cand, tool, secant_iters);
    interact32_block<kFused, kB, kStaged, kMlp, kSplit>(blockIdx.x, N, K, offsets, rec, cand, B, F, seg, tool,
                                                        secant_iters, status, cap, mlp);
}

template <int kB, int kMinB, bool kStaged, bool kMlp = false, int kSplit = 1>
static void launch_i32(cudaStream_t s, int N, const KConsts &K, const int32_t *offsets, const SortedFields32 &B,
                       const FixedFields32 &F, const StepScratch &W, const SegDev &seg, const ToolDev *tool, int cap,
                       const MlpDev &mlp = MlpDev{}) {
    size_t smem = 0;
    if (kStaged) {
        smem = (size_t)cap * 64 + sizeof(int) * (kChunk32 + 1) * kB;
        static bool configured = false;   // opt in above 48 KB of dynamic shared memory, once
        if (!configured) {
            cudaFuncSetAttribute(k_interact32<true, kB, kMinB, kStaged, kMlp, kSplit>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            configured = true;
        }
    }
    launch_after(s, k_interact32<true, kB, kMinB, kStaged, kMlp, kSplit>, div_up(N, kB / kSplit), kB, smem, N, K, offsets,
                 W.rec32, W.cand32, B, F, seg, tool, W.secant_iters, W.status, cap, mlp);
}

// The default shape on grids of few waves: no bound on the registers (95 instead of 79,
// five blocks an SM instead of six), so that the loads of a pair and of the epilogue are
// issued further ahead -- where a wave of five takes no more waves than one of six, by more
// than a scrap of the last one, and up to three.  Steps, six blocks -> five (152 SMs, waves
// of 116,736 and 97,280 particles): 12,000 particles (cut) 71.1 -> 68.9 us; lattices 90,000
// 63.6 -> 59.8, 160,000 97.9 -> 94.4, 193,600 106.2 -> 100.5, 250,000 132.5 -> 129.7, 291,600
// 148.9 -> 144.3; but with a wave more 99,225 69.0 -> 74.2, 105,625 71.3 -> 78.8, 202,500 111.0 ->
// 113.4, 230,400 116.9 -> 120.6, 313,600 157.8 -> 159.5, 422,500 204.6 -> 206.3, and just past a
// whole wave of six 119,025 82.1 -> 82.3, 235,225 125.6 -> 127.1.  The sums are the same; as
// between all shapes, the compiler may fuse a multiply-add of the epilogue differently.
// With the warm start in the epilogue (kMlp) the unbounded shape takes 193 registers, two
// blocks an SM: on grids of one such wave, 12,000 particles (cut) 78.5 -> 75.5 us, 22,500
// (lattice) 57.4 -> 54.8; but 40,000 58.7 -> 69.0, 90,000 77.5 -> 112.2, 291,600 190 -> 284.
template <bool kMlp>
inline bool few_waves32(int N) {
    if (kMlp) return N <= 2 * sm_count() * 128;
    const int five = 5 * sm_count() * 128, six = 6 * sm_count() * 128;
    return N <= 3 * five && div_up(N, five) == div_up(N, six) && (N <= five || (N - 1) % six >= six / 8);
}

// The launch shapes of kInteractVariants (interactions.cu), in its order.
template <bool kMlp>
void launch_i32_variant(cudaStream_t s, int N, const KConsts &K, const int32_t *offsets, const SortedFields32 &B,
                        const FixedFields32 &F, const StepScratch &W, const SegDev &seg, const ToolDev *tool,
                        int variant, const MlpDev &mlp) {
    switch (variant) {
        case 1: launch_i32<64, 12, false, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 0, mlp); break;
        case 2: launch_i32<64, 8, false, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 0, mlp); break;
        case 3: launch_i32<128, 4, false, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 0, mlp); break;
        case 4: launch_i32<256, 3, false, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 0, mlp); break;
        case 5: launch_i32<256, 1, false, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 0, mlp); break;
        case 6: launch_i32<128, 3, true, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 640, mlp); break;
        case 7: launch_i32<128, 2, true, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 1024, mlp); break;
        case 8: launch_i32<64, 6, true, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 384, mlp); break;
        case 9: launch_i32<256, 2, true, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 1024, mlp); break;
        case 10: launch_i32<128, 6, false, kMlp, 2>(s, N, K, offsets, B, F, W, seg, tool, 0, mlp); break;
        case 11: launch_i32<128, 6, false, kMlp, 4>(s, N, K, offsets, B, F, W, seg, tool, 0, mlp); break;
        case 12: launch_i32<128, 5, false, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 0, mlp); break;
        case 13: launch_i32<64, 10, false, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 0, mlp); break;
        default:
            if (few_waves32<kMlp>(N)) launch_i32<128, 1, false, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 0, mlp);
            else launch_i32<128, 6, false, kMlp>(s, N, K, offsets, B, F, W, seg, tool, 0, mlp);
            break;
    }
}

}  // namespace sphfem
