// state.cuh -- device-side layout of the particle state and step scratch.
#pragma once

#include "common.cuh"

namespace sphfem {

// The 20 fields reordered by the Green sort (grid_gpu_green.cu:55-113) plus
// the sort keys; two copies, swapped after each sort like the reference.
struct SortedFields {
    double2 *pos, *vel, *fc, *ft, *n;
    double *h, *rho, *eps_pl, *eps_pl_dot, *T, *fixed, *blanked, *tool_particle;
    dbl4 *S;
    double2 *pos_t, *vel_t;
    double *rho_t, *T_t;
    dbl4 *S_t;
    int32_t *on_seg;
    int32_t *hash;
};

// The same fields in the compact form of FP32K contexts: positions and density
// in FP64 (the corrector's x + dt*x_t and rho + dt*rho_t, where FP32 would lose
// the small increments), everything else in FP32; the 0/1 flags as floats.
// 148 bytes per particle instead of 284.  Every value the FP32K step computes
// for these fields is an FP32 value already, so storing them in FP32 changes
// no result of the step except the contact forces and normals, which the
// contact search still computes in FP64 and now rounds once to FP32.
struct SortedFields32 {
    double2 *pos;
    float2 *vel, *fc, *ft, *n;
    float *h;
    double *rho;
    float *eps_pl, *eps_pl_dot, *T, *fixed, *blanked, *tool_particle;
    float4 *S;
    float2 *pos_t, *vel_t;
    float *rho_t, *T_t;
    float4 *S_t;
    int32_t *on_seg;
    int32_t *hash;
};

// Arrays that are not reordered by the sort (particle_gpu fields the Green
// buffer does not carry: p, R, S_der, v_der, idx).
struct FixedFields {
    double *p;
    dbl4 *R;
    dbl4 *S_der, *v_der;
    int32_t *idx;
};

// p and R of the FP32K step (R.w unused); S_der, v_der and idx stay in FixedFields.
struct FixedFields32 {
    float *p;
    float4 *R;
};

// Scratch of the counting sort.
struct SortScratch {
    int32_t *key;        // [N] sort key of each particle (hash, or num_cell when out of range)
    int32_t *hash_next;  // [N] raw hash taken by the histogram pass (the fused step keeps the
                         //     visible hash array as the reference leaves it until the next sort)
    int32_t *arrival;    // [N] arrival slot inside its cell (atomic counter value)
    int32_t *counts;     // [num_cell+1] particles per cell (last = out-of-grid bucket), then the contact queue's length
    int32_t *offsets;    // [num_cell+2] exclusive scan of counts
    int32_t *slots;      // [N] particle ids grouped by cell, arbitrary order inside a cell; the tail's contact queue
    int32_t *block_sums; // scan partials
    int32_t *cell_start, *cell_end;   // grid_gpu_green m_cell_start / m_cell_end
};

// Packed neighbour record: what a neighbour contributes to the pair sums.
// FP64: 16 doubles = 128 B; FP32K: 16 floats = 64 B (positions as offsets
// from the particle's cell corner; the last word packs the cell row and flags).
constexpr int kRecWords = 16;
// kFlagNonFinite: a value of an active particle's record is NaN or infinite
// (its pair terms are NaN even with the zero kernel weights outside the
// support); never set on blanked records.
// kFlagFar (FP32 records): the position is so far from its cell's box (moved since
// the sort) that its candidate entry cannot stand for it.
enum : int {
    kFlagFar = (int)0x80000000u, kFlagBlanked = 1 << 30, kFlagTool = 1 << 29, kFlagNonFinite = 1 << 28,
    kRowMask = (1 << 28) - 1
};

// An FP32 record's four quarters lie in four arrays: the lanes of a warp read
// neighbours that are mostly near one another in cell order, and with eight quarters
// to a 128-byte line a pass of the L1 serves more lanes than with two whole records --
// the neighbour sums are bound by these passes (2,640 a warp with whole records read
// by 256-bit loads, 2,250 with halves, 2,060 with quarters).
__device__ __forceinline__ void put_rec32(float4 *__restrict__ rec, int N, int k, float4 r0, float4 r1, float4 r2,
                                          float4 r3) {
    rec[k] = r0;
    rec[(size_t)N + k] = r1;
    rec[2 * (size_t)N + k] = r2;
    rec[3 * (size_t)N + k] = r3;
}

// FP32 candidate entry, one float2 per record in the same order, for the in-support
// test of the candidate scan: (x - x_cell, y8), 8 bytes instead of the record's first
// 16.  y8 is the y coordinate in a frame that repeats every 8 cells, (row mod 8) cell +
// (y - y_cell): rows that a stencil joins are at most 3 apart, so min(|d|, 8 cell -
// |d|) of two entries' difference d is their distance in y, with no row to decode.  y8
// is below 8 cells: its rounding moves the test's boundary by less than 2^-19 of a cell,
// where the kernel and its gradient vanish to third and second order; the pair terms
// use the full record.  A blanked record's entry fails every test (x infinite); one
// whose record is marked non-finite or far passes every test (x NaN, in a test that
// NaN passes), and the record's flags decide.
__device__ __forceinline__ float cand_y8(float yr, int row, float cell) { return fmaf((float)(row & 7), cell, yr); }
__device__ __forceinline__ int cand_far(float xr, float yr, float cell) {
    return fabsf(xr - 0.5f * cell) <= 0.75f * cell && fabsf(yr - 0.5f * cell) <= 0.75f * cell ? 0 : kFlagFar;
}
__device__ __forceinline__ float2 cand_pack32(float xr, float yr, int flags, float cell) {
    const float x = (flags & kFlagBlanked) ? __int_as_float(0x7f800000)
                    : (flags & (kFlagNonFinite | kFlagFar)) ? __int_as_float(0x7fffffff) : xr;
    return make_float2(x, cand_y8(yr, flags & 7, cell));
}

// Per-segment constants of the contact search, rebuilt each step with the
// y-bins (k_seg_bins), after the tool has moved: what on_segment_mesh and the
// first loop of find_shortest_distance_v1 (actions_gpu.cu:51-63, :139-180)
// form per particle from the segment alone, computed once with the same
// operations -- so every test gives the reference's result bit for bit.
struct __align__(64) SegGeo {
    long long kx0, kx1, ky0, ky1;     // order keys of xmin - 0.0008, xmax + 0.0008, ymin - 0.0008, ymax + 0.0008
    double ymin_f, ymax_f;            // fminf / fmaxf of the end points' y (float-rounded)
    double inv_slope;                 // (left.x - right.x) / (left.y - right.y), non-horizontal segments
    long long pad;
};

// Interface segments (segment_FEM_gpu, segment_FEM_gpu.h:31-56).
struct SegDev {
    int n;
    double2 *left, *right, *normal;
    int4 *marks;              // element, colour, node left, node right
    double2 *heat_exchange;   // (sum T*length, sum length)
    double *fric_heat;
    double2 *robin;           // fused step: each segment's Robin terms (rhs, diagonal) for its two nodes
    WearAcc wear;             // wear statistics (pp == NULL: off)
    double *wear_rate;        // wear_nodes: per-segment wear rate of the last nodal shift
    // y-bins of each case's segments for the contact's ray casting (k_seg_bins):
    // bin_count[case * kSegBins + b] segments listed, -1 when the bin overflowed
    // (then the full scan runs); bin_list[(case * kSegBins + b) * kSegBinCap + k]
    // the case-local segment index.  NULL: no bins, full scan.
    int32_t *bin_count;
    int32_t *bin_list;
    // with the bins: per segment, SegGeo; per bin, the order key of an x bound
    // right of which no segment of the bin has a crossing (an empty bin: the
    // lowest key)
    SegGeo *geo;
    long long *bin_xkey;
};
constexpr int kSegBins = 64;
constexpr int kSegBinCap = 256;

// FEM thermal system of the tool (FEM_thermal_2D_GPU, FEM_thermal_gpu.h:35-93).
// K, f are the assembled (post-Dirichlet) m_stiffness_matrix / m_f; the Robin
// terms of apply_robin_bdc are added on the fly from the segments touching a
// node (node_seg_ptr / node_seg), so no K_temp/f_temp copy is made per step.
struct FemDev {
    int n_nodes, nnz;
    double2 *position;
    int32_t *row_ptr, *col_ind, *diag;   // diag[i] = CSR slot of (i,i)
    double *K, *M_inv, *f, *T, *k;
    double *T_half;                      // T after calculate_temp(0.5 dt)
    int32_t *node_seg_ptr, *node_seg;    // segments whose left/right node is this node
    double *M;                           // lumped mass (m_mass_matrix); allocated with wear only
};

// Wear by nodal shift: the nodes of the two cutting-edge layers, each with its
// layer elements (x: element, y: the node's local index) and the CSR slots of
// (node, element node b), b = 0..2, for the atomic-free retreat / resume of the
// layers' mass and stiffness; the per-segment node shifts; the wear constants.
struct WearDev {
    int n_elem;                          // layer elements
    const int32_t *elem;                 // [n_elem] element ids
    double *mat_old, *mat_new;           // [n_elem][10]: lumped mass, stiffness (row-major) before / after the shift
    int n_nodes;                         // nodes of layer elements
    const int32_t *node;                 // [n_nodes] node ids
    const int32_t *adj_ptr;              // [n_nodes + 1]
    const int4 *adj;                     // (layer element index, local index)
    const int4 *slot;                    // CSR slots (x, y, z)
    const int4 *elements;                // [n_elements] node a, b, c, colour
    dbl4 *seg_delta;                     // [n_seg] shift of the left (x, y) and right (z, w) node
    double A, B, C, D;                   // wear constants (constants_structs.h:113-119)
};

// Candidate entry beside the FP64 records, for a test that only sorts out candidates
// that cannot be in the support: (x - x_cell, y - y_cell), the flags in the low
// mantissa bits: x's two lowest hold kCandBlanked / kCandSpecial, y's three lowest the
// cell row modulo 8.  kCandSpecial marks the ones that the test may not sort out -- a
// non-finite record, or coordinates further than 4 cells from the cell (positions
// moved since the sort), where FP32 is too coarse.
enum : int { kCandBlanked = 1, kCandSpecial = 2 };
__device__ __forceinline__ float2 cand_pack64(float xr, float yr, float cell, int flags) {
    const bool near = fabsf(xr) <= 4.f * cell && fabsf(yr) <= 4.f * cell;
    const int bx = (__float_as_int(xr) & ~3) | ((flags & kFlagBlanked) ? kCandBlanked : 0) |
                   (!near || (flags & kFlagNonFinite) ? kCandSpecial : 0);
    const int by = (__float_as_int(yr) & ~7) | (flags & 7);
    return make_float2(__int_as_float(bx), __int_as_float(by));
}

struct StepScratch {
    dbl4 *rec64;      // [N][4] FP64 records
    float4 *rec32;       // [4][N] FP32 records, quarter by quarter (put_rec32)
    float2 *cand32;      // [N, padded to whole groups of 4] candidate entries of the records (cand_pack32, cand_pack64)
    double2 *pos_init, *vel_init;   // leap_frog snapshots (staged path)
    dbl4 *S_init;
    double *rho_init, *T_init;
    int32_t *secant_iters;          // [N] secant iterations of the last JC pass (0 = elastic)
    uint32_t *status;               // device status word
    double *reduce;                 // reduction scratch
};

// The learned warm start of the return mapping: a 4-64-64-64-1 SiLU MLP.
// Parameters in FP32 (layout kMlp* offsets); BF16 copies of the four weight
// matrices feed the tensor cores.  Features and target are standardised with
// the training set's moments.
constexpr int kMlpIn = 4, kMlpH = 64;
constexpr int kMlpOffW1 = 0, kMlpOffB1 = 256, kMlpOffW2 = 320, kMlpOffB2 = 4416, kMlpOffW3 = 4480,
              kMlpOffB3 = 8576, kMlpOffW4 = 8640, kMlpOffB4 = 8704, kMlpParams = 8705;
// BF16 weight copies: W1 [64][4], W2 [64][64], W3 [64][64], W4 [64]
constexpr int kMlpWbW1 = 0, kMlpWbW2 = 256, kMlpWbW3 = 4352, kMlpWbW4 = 8448, kMlpWb = 8512;

struct MlpDev {
    const float *params;      // [kMlpParams] FP32 (biases are read from here)
    const uint16_t *wb;       // [kMlpWb] BF16 bit patterns of the weights
    float x_mean[4], x_inv_std[4], y_mean, y_std;
};

}  // namespace sphfem
