// interact64.cuh -- the FP64 neighbour sums (k_interact64) and their fused
// epilogue; included by interactions.cu, whose header describes the sums.
//
// Bound: the FP64 pipe, two operations per SM and clock.  One thread per particle
// with every operation in FP64 took 4,872 FP64 instructions per 32 particles on the
// lattice of 2h cells and kept the pipe 87 % busy; this kernel takes 1,400 (67 % of
// a launch of 262,144 particles):
//  * candidates are tested in FP32 on the 8-byte entries with a margin that no
//    in-support neighbour can fall outside of; the FP64 test then runs only on
//    the ones that pass;
//  * the pair terms that are products, quotients and polynomials of known sign --
//    the spline and its gradient over r, 1 / (rho_i + rho_j), the viscosity's
//    quotient, (W / W(dp))^4 -- run on 64-bit mantissas on the integer pipes
//    (fix64.cuh).  35 FP64 operations a pair are left, sums and differences;
//  * kLanes64 consecutive lanes share a particle and its list of neighbours, so a
//    system of a few thousand particles fills the schedulers, and the epilogue
//    runs once per particle in full warps from partial sums in shared memory.
// Neighbour stage, before and after: 1,048,576-particle lattice (2h cells) 9.40 ->
// 2.94 ms; 640,000-particle cut (cells of h) 5.53 -> 1.82 ms; 12,000-particle cut
// 0.247 -> 0.069 ms, the return mapping of the yielding particles (return_map) included.
// A particle with anything the mantissa forms do not take (a candidate marked
// non-finite, a smoothing length, density or volume outside 2^+-64, a product of
// relative velocity and distance that is subnormal or 2^300 and more) repeats its
// sums in plain FP64 over every active candidate, with the reference's zero
// weights outside the support (interactions_gpu.cu:230-337).
#pragma once

#include "fix64.cuh"
#include "interact32.cuh"

namespace sphfem {

// A quarter of a record, which nothing writes while the sums run.  (Not volatile: the compiler
// places it as it does its own loads.)
__device__ __forceinline__ dbl4 ld_nc(const dbl4 *p) {
    dbl4 v;
    asm("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}

constexpr int kLanes64 = 4;                            // lanes per particle
constexpr int kThreads64 = 128;                        // threads per block
constexpr int kParts64 = kThreads64 / kLanes64;        // particles per block
constexpr int kList64 = 64, kListPitch64 = kList64 + 4;   // neighbours per pass; the pitch spreads a warp's lists over the banks

// |x| < 2^500: with such viscosity constants and (v, x) below 2^300 no product overflows.
__device__ __forceinline__ bool below_2_500(double x) { return ((uint32_t)__double2hiint(x) & 0x7fffffffu) < 0x5f300000u; }

// v_der, S_der / mass, vel_t / (-mass), pos_t / (eps mass), T_lapl / 2
struct Sums64 {
    double vd0, vd1, vd2, vd3, sd0, sd1, sd2, sd3, vt0, vt1, xt0, xt1, tl;
};

// Plain FP64 sums over every active candidate j = first, first + kLanes64, ... of
// the stencil's columns (the reference's body with cubic_spline's zero weights,
// kernels.cuh:37-39).
static __device__ __noinline__ void sums64_plain(Sums64 &out, int k, int sub, const int32_t *__restrict__ offsets,
                                          const dbl4 *__restrict__ rec, int hash, int nx, int ny, int R, double inv_wdp,
                                          double eta2, double beta, bool tool_i, bool thermal) {
    const dbl4 i0 = rec[4 * k + 0], i1 = rec[4 * k + 1], i2 = rec[4 * k + 2], i3 = rec[4 * k + 3];
    const double hi = i2.z;
    const double h1 = 1 / hi, fourh2 = 4 * hi * hi, fac = kPiFac * h1 * h1;
    const int gi = hash / ny, gj = hash - gi * ny;
    Sums64 a = {};
    for (int ii = max(gi - R, 0); ii < min(gi + R + 1, nx); ii++) {
        const int j1 = __ldg(offsets + ii * ny + min(gj + R + 1, ny));
        for (int j = __ldg(offsets + ii * ny + max(gj - R, 0)) + sub; j < j1; j += kLanes64) {
            const dbl4 n0 = rec[4 * j + 0], n1 = rec[4 * j + 1], n2 = rec[4 * j + 2], n3 = rec[4 * j + 3];
            const int fj = (int)__double_as_longlong(n3.w);
            if (fj & kFlagBlanked) continue;
            const double dx = i0.x - n0.x, dy = i0.y - n0.y;
            const double rr2 = dx * dx + dy * dy;
            const double rad = sqrtf_d(rr2);
            const double q = rad * h1;
            double val, der;
            if (q > 1) {
                const double t = 2 - q, t2 = t * t;
                val = 0.25 * t2 * t2 * t2;
                der = -0.75 * t2 * h1 / rad;
            } else {
                val = 1 - 1.5 * q * q * (1 - 0.5 * q);
                der = -3.0 * q * (1 - 0.75 * q) * h1 / rad;
            }
            const bool zero_w = rr2 >= fourh2 || rr2 < 1e-8;
            const double w = zero_w ? 0. : val * fac;
            const double dwf = zero_w ? 0. : der * fac;
            const double wx = dwf * dx, wy = dwf * dy;
            const double volj = n3.y;
            if (!tool_i && !(fj & kFlagTool)) {
                const double dvx = n0.z - i0.z, dvy = n0.w - i0.w;
                const double tx = wx * volj, ty = wy * volj;
                a.vd0 += dvx * tx;
                a.vd1 += dvx * ty;
                a.vd2 += dvy * tx;
                a.vd3 += dvy * ty;
                double fab = w * inv_wdp;
                fab *= fab;
                fab *= fab;
                const double ax = (i1.x + n1.x) + fab * (i1.w + n1.w);
                const double ay = (i1.y + n1.y) + fab * (i2.x + n2.x);
                const double az = (i1.z + n1.z) + fab * (i2.y + n2.y);
                a.sd0 += ax * wx;
                a.sd1 += ay * wy;
                a.sd2 += ay * wx;
                a.sd3 += az * wy;
                const double vijposij = -(dvx * dx + dvy * dy);
                const double irho = 1. / (0.5 * (i2.w + n2.w));
                if (vijposij < 0.) {
                    const double hij = 0.5 * (hi + n2.z);
                    const double muij = (hij * vijposij) / (rr2 + eta2 * hij * hij);
                    const double piij = ((i3.x + n3.x) * muij + beta * muij * muij) * irho;
                    a.vt0 += piij * wx;
                    a.vt1 += piij * wy;
                }
                const double wr = w * irho;
                a.xt0 += wr * dvx;
                a.xt1 += wr * dvy;
            }
            // Brookshaw, (e.dW)/r == dW/dr; the reference skips it at r <= 1e-8 (interactions_gpu.cu:328)
            if (thermal && (!zero_w || rr2 > 1e-16)) a.tl += volj * (i3.z - n3.z) * dwf;
        }
    }
    out = a;
}

// ---- per-particle epilogue (fused mode) -----------------------------------------------------------
// vd (= v_der), acc (stress divergence and viscosity, an acceleration), xt (= pos_t from XSPH), T_t.
// Returns whether the particle may yield: return_map then finishes it.
__device__ __forceinline__ bool fused_epilogue(int k, const KConsts &K, const SortedFields &B, const FixedFields &F,
                                               const SegDev &seg, const ToolDev *__restrict__ tool,
                                               int32_t *__restrict__ secant_iters, uint32_t *status, bool is_tool,
                                               double2 vel_pred, double rho_pred, dbl4 vd, double2 acc, double2 xt,
                                               bool thermal, double T_t_new) {
    const ToolDev &tc = tool[case_of_hash(K, B.hash[k])];   // the particle's case (time step, tool)
    const double dt = tc.dt;
    const double mass = K.c.phys.mass;
    dbl4 S0 = B.S[k];
    dbl4 St = B.S_t[k];
    double2 pos_t, vel_t;
    double rho_t = B.rho_t[k];
    if (!is_tool) {
        const double hdt = 0.5 * dt;
        dbl4 Sp = mk4(S0.x + hdt * St.x, S0.y + hdt * St.y, S0.z + hdt * St.z, S0.w + hdt * St.w);
        St = jaumann_one(K, vd, Sp);                                  // actions_gpu.cu:280-314
        rho_t = -rho_pred * (vd.x + vd.w);                            // actions_gpu.cu:626-639
        const double2 fc = B.fc[k], ft = B.ft[k];
        vel_t = acc;                                                  // actions_gpu.cu:641-671
        // no division for the particles without a contact force: adding 0 / mass changes nothing
        if (flag_nonzero(fc.x) || flag_nonzero(ft.x)) vel_t.x += fc.x / mass + ft.x / mass;
        if (flag_nonzero(fc.y) || flag_nonzero(ft.y)) vel_t.y += fc.y / mass + ft.y / mass;
        pos_t.x = xt.x + vel_pred.x;                                  // actions_gpu.cu:673-687
        pos_t.y = xt.y + vel_pred.y;
    } else if (K.thermal_pse) {   // PSE build: tool particles leave the sums unwritten
        vel_t = B.vel_t[k];
        pos_t = B.pos_t[k];
    } else {
        vel_t = acc;
        pos_t = xt;
    }
    double T_t = thermal ? T_t_new : B.T_t[k];
    B.pos_t[k] = pos_t;
    B.vel_t[k] = vel_t;
    B.S_t[k] = St;
    B.rho_t[k] = rho_t;
    B.T_t[k] = T_t;
    // correct (leap_frog.cu:71-96)
    double2 pos = B.pos[k], vel = B.vel[k];
    pos.x = pos.x + dt * pos_t.x;
    pos.y = pos.y + dt * pos_t.y;
    vel.x = vel.x + dt * vel_t.x;
    vel.y = vel.y + dt * vel_t.y;
    dbl4 S = mk4(S0.x + dt * St.x, S0.y + dt * St.y, S0.z + dt * St.z, S0.w + dt * St.w);
    double rho = B.rho[k] + dt * rho_t;
    double T = B.T[k] + dt * T_t;
    B.pos[k] = pos;
    B.vel[k] = vel;
    B.rho[k] = rho;
    double blanked = 0.;
    uint32_t st = 0;
    // friction heat (actions_gpu.cu:345-420), tool runs only
    if (K.has_tool) st |= fric_heat_one(K, dt, tc.vel, vel, B.ft[k], B.n[k], B.fc[k], rho, B.eps_pl[k], B.on_seg[k],
                                        seg.n, T, blanked, seg.fric_heat, seg.wear);
    else if (K.rigid && !is_tool && K.c.trml_wp.eta != 0.)   // actions_gpu.cu:316-343
        rigid_fric_heat_one(K, dt, K.rigid->vel, vel, B.ft[k], B.n[k], T);
    bool yields = false;
    if (K.c.plastic && !is_tool && blanked != 1.) {   // return mapping (actions_gpu.cu:689-754)
        yields = !surely_elastic(K, S, F.p[k], B.eps_pl[k], B.eps_pl_dot[k], T);
        if (!yields) {
            B.eps_pl_dot[k] = 0.;
            if (secant_iters) secant_iters[k] = 0;
        }
    }
    B.S[k] = S;
    B.T[k] = T;
    if (blanked == 1.) B.blanked[k] = 1.;
    if (st) set_status(status, st);
    return yields;
}

// The return mapping of a particle that may yield, from its stored state, by one lane or
// four (return_mapping).  Not inlined: with its code in the kernel's own the sums of
// 1,048,576 particles take 2,917 us, so 2,883.
template <bool kQuad>
static __device__ __noinline__ void return_map(int k, const KConsts &K, const SortedFields &B, const double *p,
                                               const ToolDev *tool, int32_t *secant_iters, uint32_t *status) {
    dbl4 S = B.S[k];
    double T = B.T[k], blanked = 0.;
    Mapping64 y;
    y.eps_pl = B.eps_pl[k];
    y.eps_pl_dot = B.eps_pl_dot[k];
    y.T = T;
    y.dt = tool[case_of_hash(K, B.hash[k])].dt;
    trial_norms(S, p[k], y.norm, y.svm);
    const Mapped64 m = return_mapping<kQuad>(K, y);
    if (kQuad && (threadIdx.x & 3u)) return;
    B.eps_pl_dot[k] = m.eps_pl_dot;
    if (secant_iters) secant_iters[k] = abs(m.iters);
    if (m.iters == 0) return;   // elastic after all
    B.eps_pl[k] = m.eps_pl;
    const uint32_t st = apply_mapping(K, y, m, B.rho[k], S, T, blanked);
    B.S[k] = S;
    B.T[k] = T;
    if (blanked == 1.) B.blanked[k] = 1.;
    if (st) set_status(status, st);
}

// ---- the kernel --------------------------------------------------------------------------------------
// kMapNone: the staged sums.  kMapLane, kMapQuads: the fused step, its return mappings in
// the epilogue's lanes or in groups of four lanes of the whole block.  The groups cut a
// small system's step, whose last block waits for one chain (12,000 particles, 74 of them
// yielding, sums stage 81 -> 72 us), but keep the block's other warps, and their registers,
// until the epilogue's end: on systems of many waves, where the next block's warps would
// start in their place, 2 % slower (1,048,576 particles 2,891 -> 2,949 us).  So: groups on
// grids of up to one wave (map_by_quads).
enum Map64 { kMapNone, kMapLane, kMapQuads };
inline bool map_by_quads(int N) { return div_up(N, kParts64) <= 5 * sm_count(); }
// kBlocks: blocks an SM that the registers must leave room for.  5 (20 warps, 96
// registers, 164 bytes spilled) on a grid of many waves, where warps alternate between the
// integer and the FP64 pipe: 4 blocks at 128 registers were 5 % slower on the
// 1,048,576-particle lattice, 3 blocks 13 %.  3, with 156 registers and nothing spilled, on
// a grid that needs no more (three_blocks): step of 12,000 particles (cut) 112.2 -> 107.4 us,
// of 7,355 (rigid, PSE) 93.2 -> 89.4, of 1,600 (lattice) 58.5 -> 53.3; but of 19,600 99.6 ->
// 117.4.
inline bool three_blocks(int N) { return div_up(N, kParts64) <= 3 * sm_count(); }
template <Map64 kMap>
__device__ __forceinline__ void interact64_block(int N, const KConsts &K, const int32_t *__restrict__ offsets,
                                                 const dbl4 *__restrict__ rec, const float2 *__restrict__ cand,
                                                 const SortedFields &B, const FixedFields &F, const SegDev &seg,
                                                 const ToolDev *__restrict__ tool, int32_t *__restrict__ secant_iters,
                                                 uint32_t *status) {
    constexpr bool kFused = kMap != kMapNone;
    constexpr int kSums = kFused ? 9 : 13;
    __shared__ int s_list[kParts64 * kListPitch64];
    __shared__ double s_sum[kSums][kThreads64];
    const int sub = (int)threadIdx.x % kLanes64, part = (int)threadIdx.x / kLanes64;
    const int lane = (int)threadIdx.x & 31;
    const unsigned gshift = (unsigned)(lane & ~(kLanes64 - 1));
    const int k = (int)blockIdx.x * kParts64 + part;
    int *list = s_list + part * kListPitch64;
    const int kk = min(k, N - 1);
    const dbl4 i0 = ld_nc(rec + 4 * kk), i1 = ld_nc(rec + 4 * kk + 1), i2 = ld_nc(rec + 4 * kk + 2),
               i3 = ld_nc(rec + 4 * kk + 3);
    const int fi = (int)__double_as_longlong(i3.w);
    const int hash = B.hash[kk];
    const sph_geom_constants &geo = K.g;
    const bool tool_i = (fi & kFlagTool) != 0;
    // PSE build: tool particles return at once
    const bool live = k < N && !(fi & kFlagBlanked) && hash >= 0 && hash < geo.num_cell && !(K.thermal_pse && tool_i);
    const double xi = i0.x, yi = i0.y, hi = i2.z;
    const double thermal_alpha = (!tool_i) ? K.c.trml_wp.alpha : K.c.trml_tool_sph.alpha;
    const bool thermal = flag_nonzero(thermal_alpha) && !K.thermal_pse;   // Brookshaw build only
    double fourh2 = 4 * hi * hi;
    double eta2h2 = K.eta2 * 0.25 * fourh2;
    // kept in registers (or spilled): the compiler otherwise forms them again for every pair
    asm volatile("" : "+d"(fourh2), "+d"(eta2h2));

    // Per-particle constants of the spline with W = fac w(q), q = r / h:
    // q > 1: w = (2-q)^6 / 4, dW/(r dr) = -3/4 fac h1 (2-q)^2 / r;
    // q <= 1: w = 1 - 3/2 q^2 + 3/4 q^3, dW/(r dr) = -3 fac h1^2 (1 - 3/4 q).
    bool plain = !fix_range(hi) || !fix_range(K.inv_wdeltap) || !fix_range(fourh2 + eta2h2) ||
                 !below_2_500(K.c.corr.alpha) || !below_2_500(K.c.corr.beta) || (fi & kFlagNonFinite);
    const double h_safe = plain ? 1. : hi;
    const Fix64 h1 = fix_recip_rn(h_safe), hm = fix_of(h_safe);
    const Fix64 fac = fix_norm(fix_of(kPiFac) * (h1 * h1));
    const Fix64 c_far = fix_norm(fix_of(0.75) * (fac * h1)), c_near = fix_norm(fix_of(3.) * (fac * (h1 * h1)));
    const Fix64 iwdp = fix_of(plain ? 1. : K.inv_wdeltap);

    double vd0 = 0, vd1 = 0, vd2 = 0, vd3 = 0, sd0 = 0, sd1 = 0, sd2 = 0, sd3 = 0, vt0 = 0, vt1 = 0, xt0 = 0, xt1 = 0,
           tl = 0;   // fused: sd0, sd2 hold the acceleration / mass; sd1, sd3, vt0, vt1 unused

    const int gi = live ? hash / geo.ny : 0, gj = live ? hash - gi * geo.ny : 0, R = geo.stencil;
    int ii = live ? max(gi - R, 0) : 0;
    const int ii1 = live ? min(gi + R + 1, geo.nx) : 0;
    const int lo_j = max(gj - R, 0), hi_j = min(gj + R + 1, geo.ny);
    const float2 ce = live ? cand[kk] : make_float2(0.f, 0.f);
    const float cell = K.f.cell;
    // The candidate test's margin: an entry's coordinates lie within 4 cells (cand_pack64
    // marks the others), so they and the FP32 arithmetic are off by less than 2^-16 cell
    // <= 2^-12 h; rr2 by less than 1e-3 h^2 of the 4 h^2 compared with.
    const float limit = 4.008f * float_trunc(hi) * float_trunc(hi);
    const bool take_all = (__float_as_int(ce.x) & kCandSpecial) || !(cell <= 16.f * float_trunc(hi));
    int j = 0, j1 = 0;
    if (ii < ii1) {
        j = __ldg(offsets + ii * geo.ny + lo_j);
        j1 = __ldg(offsets + ii * geo.ny + hi_j);
    }
    bool done = ii >= ii1;
    while (true) {
        // phase 1: the group's list of candidates that may be in the support, kLanes64 at a time
        int cnt = 0;
        while (true) {
            while (!done && j >= j1) {   // the next column with candidates
                if (++ii >= ii1) {
                    done = true;
                } else {
                    j = __ldg(offsets + ii * geo.ny + lo_j);
                    j1 = __ldg(offsets + ii * geo.ny + hi_j);
                }
            }
            const bool more = !done && cnt <= kList64 - kLanes64;
            if (!__any_sync(0xffffffffu, more)) break;
            bool take = false;
            const int jj = j + sub;
            if (more && jj < j1) {
                const float2 c = __ldg(cand + jj);
                const float dx = (float)(gi - ii) * cell + (ce.x - c.x);
                const float dy = (float)cand_row_diff(gj, c.y) * cell + (ce.y - c.y);
                take = (dx * dx + dy * dy < limit && jj != k) || take_all || (__float_as_int(c.x) & kCandSpecial);
                take = take && !(__float_as_int(c.x) & kCandBlanked);
            }
            const unsigned takes = (__ballot_sync(0xffffffffu, take) >> gshift) & ((1u << kLanes64) - 1u);
            if (take) list[cnt + __popc(takes & ((1u << sub) - 1u))] = jj;
            cnt += __popc(takes);
            if (more) j += kLanes64;
        }
        __syncwarp();
        // phase 2: the pair body over the list, shared by the group's lanes
        for (int t = sub; t < cnt; t += kLanes64) {
            const int jn = list[t];
            const dbl4 n0 = ld_nc(rec + 4 * jn), n1 = ld_nc(rec + 4 * jn + 1), n2 = ld_nc(rec + 4 * jn + 2),
                       n3 = ld_nc(rec + 4 * jn + 3);
            const int fj = (int)__double_as_longlong(n3.w);
            const double ex = n0.x - xi, ey = n0.y - yi;   // minus the reference's distance vector
            const double rr2 = ex * ex + ey * ey;
            const double sum_rho = i2.w + n2.w;
            if ((fj & kFlagNonFinite) || !fix_range(n3.y) || !fix_range(sum_rho)) plain = true;
            const long long b2 = __double_as_longlong(rr2);
            if (plain || b2 >= __double_as_longlong(fourh2) || b2 < __double_as_longlong(1e-8)) continue;
            const float rad = sqrtf(float_of_normal(rr2));   // sqrtf of the rounded argument (kernels.cuh:45)
            // q as the reference's double: beside q = 2 its rounding is all that 2 - q holds
            const Fix64 qd = fix_mul_rn(h1, rad);
            const uint64_t q = qd.m >> min(max(-61 - qd.e, 0), 63);   // q 2^61
            const uint64_t one = 1ull << 61;
            // both branches of the spline, then a selection: the lanes stay together for
            // the FP64 instructions that follow
            const long long d = (long long)(2 * one - q);
            const Fix64 u = fix_norm({(uint64_t)(d < 0 ? -d : d), -61});
            const Fix64 u2 = u * u;
            const uint64_t q1 = q << 2, q2 = mul_hi(q1, q1), q3 = mul_hi(q2 << 1, q1);   // q <= 1: 2^63, 2^62, 2^62
            const bool far = q > one;
            Fix64 val = (u2 * u2) * u2;
            val.e -= 2;
            val.m = far ? val.m : (1ull << 62) - q2 - (q2 >> 1) + q3 - (q3 >> 2);
            val.e = far ? val.e : -62;
            Fix64 dw = c_far * fix_recip(rad);
            dw.m = far ? dw.m : c_near.m;
            dw.e = far ? dw.e : c_near.e;
            dw = dw * Fix64{far ? u2.m : (1ull << 63) - q1 + (q1 >> 2), far ? u2.e : -63};
            dw = fix_norm(dw);   // |dW/dr| / r
            const Fix64 g = fix_norm(dw * fix_of(n3.y));
            if (thermal) tl += (n3.z - i3.z) * fix_double<false>(g);
            if (tool_i || (fj & kFlagTool)) continue;
            const Fix64 w = fix_norm(val) * fac;
            const Fix64 irho = fix_recip(sum_rho);
            const double wx = fix_scale<false>(dw, ex), wy = fix_scale<false>(dw, ey);
            const double tx = fix_scale<false>(g, ex), ty = fix_scale<false>(g, ey);
            const double dvx = n0.z - i0.z, dvy = n0.w - i0.w;
            vd0 += dvx * tx;
            vd1 += dvx * ty;
            vd2 += dvy * tx;
            vd3 += dvy * ty;
            const Fix64 f1 = fix_norm(w * iwdp), f2 = f1 * f1;
            const double fab = fix_double<false>(f2 * f2);
            const Fix64 wr2 = w * irho;
            const double wr = fix_double<false>({wr2.m, wr2.e + 1});   // W / (0.5 (rho_i + rho_j))
            const double vijposij = dvx * ex + dvy * ey;
            double sxx = i1.x + n1.x, syy = i1.z + n1.z;
            const double sxy = (i1.y + n1.y) + fab * (i2.x + n2.x);
            // viscosity, for approaching pairs: mu < 0, Pi = mu (-alpha c + beta mu) / (0.5 (rho_i + rho_j))
            // -2^-1022 >= (v, x) > -2^300; a subnormal product and a diverging state's in plain FP64
            const uint32_t vh = (uint32_t)__double2hiint(vijposij);
            const bool approach = vh - 0x80100000u < 0x52a00000u;
            if (!approach && (int)vh < 0 && flag_nonzero(vijposij)) plain = true;
            Fix64 hd = hm * fix_recip(rr2 + eta2h2);   // h_ij / (r^2 + eta^2 h_ij^2)
            if (__double_as_longlong(n2.z) != __double_as_longlong(hi)) {
                // the division keeps this a branch: predicated, its FP64 operations would
                // occupy the pipe for every pair
                const double hij = 0.5 * (hi + n2.z), x = hij / (rr2 + K.eta2 * hij * hij);
                if (!fix_range(x)) plain = true;
                hd = fix_of(x);
            }
            const Fix64 mu = fix_norm(fix_norm(hd) * fix_abs(vijposij));
            const double cmu = (i3.x + n3.x) - K.c.corr.beta * fix_double<false>(mu);
            const Fix64 s1 = fix_norm(mu * irho);
            double piij = fix_scale({s1.m, s1.e + 1}, cmu, true);
            if (!approach) piij = 0.;
            if (kFused) {
                sxx -= piij;
                syy -= piij;
            }
            sxx += fab * (i1.w + n1.w);
            syy += fab * (i2.y + n2.y);
            if (kFused) {   // acceleration / mass: (stress terms - viscosity) . grad W
                sd0 += sxx * wx;
                sd0 += sxy * wy;
                sd2 += sxy * wx;
                sd2 += syy * wy;
            } else {
                sd0 += sxx * wx;
                sd1 += sxy * wy;
                sd2 += sxy * wx;
                sd3 += syy * wy;
                vt0 += piij * wx;
                vt1 += piij * wy;
            }
            xt0 += wr * dvx;
            xt1 += wr * dvy;
        }
        if (!__any_sync(0xffffffffu, !done)) break;
        __syncwarp();
    }
    const unsigned plains = (__ballot_sync(0xffffffffu, plain && live) >> gshift) & ((1u << kLanes64) - 1u);
    if (plains) {   // rare: see the head of this file
        Sums64 a;
        sums64_plain(a, k, sub, offsets, rec, hash, geo.nx, geo.ny, R, K.inv_wdeltap, K.eta2, K.c.corr.beta, tool_i, thermal);
        vd0 = a.vd0; vd1 = a.vd1; vd2 = a.vd2; vd3 = a.vd3;
        if (kFused) {
            sd0 = (a.sd0 + a.sd1) - a.vt0;
            sd2 = (a.sd2 + a.sd3) - a.vt1;
        } else {
            sd0 = a.sd0; sd1 = a.sd1; sd2 = a.sd2; sd3 = a.sd3; vt0 = a.vt0; vt1 = a.vt1;
        }
        xt0 = a.xt0; xt1 = a.xt1; tl = a.tl;
    }
    {
        double *s = &s_sum[0][threadIdx.x];
        int f = 0;
        auto put_sum = [&](double v) { s[kThreads64 * f++] = v; };
        put_sum(vd0); put_sum(vd1); put_sum(vd2); put_sum(vd3);
        put_sum(sd0);
        if (!kFused) put_sum(sd1);
        put_sum(sd2);
        if (!kFused) { put_sum(sd3); put_sum(vt0); put_sum(vt1); }
        put_sum(xt0); put_sum(xt1); put_sum(tl);
    }
    __syncthreads();
    // the epilogue, one thread per particle: a full warp for its FP64 work
    if (kMap != kMapQuads && threadIdx.x >= kParts64) return;
    const int e = (int)blockIdx.x * kParts64 + (int)threadIdx.x;
    auto particle = [&]() -> bool {
        if (e >= N) return false;
        const dbl4 e0 = ld_nc(rec + 4 * e), e2 = ld_nc(rec + 4 * e + 2), e3 = ld_nc(rec + 4 * e + 3);
        const int fe = (int)__double_as_longlong(e3.w);
        if (fe & kFlagBlanked) {
            if (kFused) rigid_heat_blanked(e, K, B);
            return false;
        }
        double v[kSums];
#pragma unroll
        for (int f = 0; f < kSums; f++) {
            const double *s = &s_sum[f][threadIdx.x * kLanes64];
            v[f] = (s[0] + s[1]) + (s[2] + s[3]);
        }
        const bool tool_e = (fe & kFlagTool) != 0;
        const double alpha_e = (!tool_e) ? K.c.trml_wp.alpha : K.c.trml_tool_sph.alpha;
        const bool thermal_e = flag_nonzero(alpha_e) && !K.thermal_pse;
        const double mass = K.c.phys.mass, xs = K.c.corr.xspheps * mass;
        const dbl4 vd = mk4(v[0], v[1], v[2], v[3]);
        const double2 xt = make_double2(xs * v[kSums - 3], xs * v[kSums - 2]);
        const double T_t = alpha_e * (2.0 * v[kSums - 1]);
        if constexpr (kFused) {
            return fused_epilogue(e, K, B, F, seg, tool, secant_iters, status, tool_e, make_double2(e0.z, e0.w), e2.w,
                                  vd, make_double2(mass * v[4], mass * v[5]), xt, thermal_e, T_t);
        } else {
            if (K.thermal_pse && tool_e) return false;
            F.S_der[e] = mk4(mass * v[4], mass * v[5], mass * v[6], mass * v[7]);
            F.v_der[e] = vd;
            B.pos_t[e] = xt;
            B.vel_t[e] = make_double2(-mass * v[8], -mass * v[9]);
            if (thermal_e) B.T_t[e] = T_t;
            return false;
        }
    };
    static_assert(kParts64 == 32, "one warp");
    if constexpr (kMap == kMapLane) {
        if (particle()) return_map<false>(e, K, B, F.p, tool, secant_iters, status);
    } else if constexpr (kMap == kMapQuads) {
        int &count = s_list[kParts64];
        if (threadIdx.x < kParts64) {
            const bool yields = particle();
            const unsigned all = __ballot_sync(0xffffffffu, yields);
            if (yields) s_list[__popc(all & ((1u << threadIdx.x) - 1u))] = e;
            if (threadIdx.x == 0) count = __popc(all);
        }
        __syncthreads();
        const int q = (int)threadIdx.x / 4;
        if (q < count) return_map<true>(s_list[q], K, B, F.p, tool, secant_iters, status);
    } else {
        particle();
    }
}

template <Map64 kMap, int kBlocks = 5>
__global__ void __launch_bounds__(kThreads64, kBlocks) k_interact64(int N, KConsts K, const int32_t *__restrict__ offsets,
                                                              const dbl4 *__restrict__ rec,
                                                              const float2 *__restrict__ cand, SortedFields B,
                                                              FixedFields F, SegDev seg,
                                                              const ToolDev *__restrict__ tool,
                                                              int32_t *__restrict__ secant_iters, uint32_t *status) {
    begin_after(offsets, rec, cand, tool, secant_iters);
    interact64_block<kMap>(N, K, offsets, rec, cand, B, F, seg, tool, secant_iters, status);
}

}  // namespace sphfem
