// Launch wrappers of the engine's CUDA kernels (sm_103a).  All pointers are
// device pointers; complex numbers are double2 (re, im); matrices are
// column-major like Eigen::MatrixXcd.  Every wrapper enqueues on `stream` and
// returns the cudaError_t of the launch.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "vdv_families.hpp"

namespace slaph {
namespace dev {

struct Q0MInst {
  int32_t t, vdv, r2;
};
struct Q1RInst {
  int32_t t, vdv, r1;
};
struct Q2MInst {
  int32_t t, b1, r1, vdv;
};
struct Q0Inst {
  int32_t t, m, r1, gamma, slot;
};
struct Q1Inst {
  int32_t t, b, r, r2, gamma, slot;
};
struct Q2Inst {
  int32_t t, b2, m, r2, gamma, slot;
};
// Q1 factors of one (Q1R, r2, b): the product that they share, and each of them.
struct X1Inst {
  int32_t t, b, r, r2;
};
struct Q1Pick {
  int32_t x, gamma, slot;  // x: instance of the batch
};
struct ProdInst {
  int32_t a, b, c;
};
struct TraceList {
  int32_t shape;
  int32_t a_base, b_base;
  int32_t stride;
  int64_t val_off;
};
struct Term {
  int32_t n;
  int32_t list[3];
  int32_t out;
  int32_t dt;
};

// Sizes every kernel needs.
struct Geometry {
  int32_t Lt, Lx, Ly, Lz, nev, dilE, n_rnd;
  int32_t nb;       // number of time-dilution blocks (Lt / dilT)
  int64_t dim_row;  // 3 * L^3
};

// Gamma table (src/Gamma.cpp:18-246) into constant memory.
// Gamma_m column c: row of its nonzero, and its value as a phase code
// (0: +1, 1: +i, 2: -1, 3: -i), for host-side planning.
int32_t gamma_row_host(int32_t m, int32_t c);
int32_t gamma_phase_host(int32_t m, int32_t c);
cudaError_t upload_gamma(cudaStream_t stream);

// One HYP smearing iteration (GaugeField::smearing_hyp, src/GaugeField.cpp:
// 322-427) of n_t consecutive timeslices of links U ([t][site][dir][9]) of a
// cubic L^3 lattice, in place; dec: scratch of n_t
// hyp_scratch_doubles_per_timeslice(L) doubles (the decorated links).
int64_t hyp_scratch_doubles_per_timeslice(int32_t L);
cudaError_t hyp_smear(double2 *U, double2 *dec, int32_t L, int32_t n_t, double alpha1,
                      double alpha2, cudaStream_t stream);
// Largest entry of a column, as it is found in pieces (norm_max.cuh): high word
// of the largest |re|, |im|, and the largest |v|^2 as the bits of a float.
struct NormMax {
  unsigned int top, n2;
};
// Displaced eigenvectors D(V_t) on a cubic lattice: n steps ((dir 0..2, forward
// 0/1) pairs, host array) with the result of the reference's in-place sweeps
// (displace_eigenvectors, src/OperatorFactory.cpp:33-55).  U: the timeslice's
// links [site][dir][a + 3 b]; P: the timeslice's line_products (read by backward
// steps only); W: scratch of nev x dim_row, twice that for n > 1.  *out: the
// result, in W, whose columns' largest entries are added to norms[nev].
// line_products: of all g.Lt timeslices, in the layout of U.
cudaError_t line_products(double2 *P, double2 const *U, Geometry g, cudaStream_t stream);
cudaError_t displaced_vectors(double2 const **out, double2 *W, double2 const *V, double2 const *U,
                              double2 const *P, int32_t const *steps, int32_t n, Geometry g,
                              cudaStream_t stream, NormMax *norms = nullptr);
// VdaggerV[2 op][t] = V_t^H W in FP64 (*op: device pointer to the operator id).
cudaError_t vdaggerv_fp64_w(double2 *vdv, double2 const *V, double2 const *W,
                            int32_t const *op, int32_t t, Geometry g, cudaStream_t stream,
                            int32_t v_t0 = 0);
// exp(-i p.x) for every op: phase[op][x] (create_momenta,
// src/OperatorFactory.cpp:64-95).  mom: [n_ops][3].
cudaError_t momenta(double2 *phase, int32_t const *mom, int32_t n_ops, Geometry g,
                    cudaStream_t stream);

// VdaggerV[vdv code 2*op][t] = V_t^H diag(e^{-ip.x}) V_t for the operators of
// the families fam[0..n_fam) (host array, vdv_families.hpp, at most kVdvFp64Ops
// operators each;
// src/OperatorFactory.cpp:292-300), FP64.  V: consecutive timeslices
// [t][nev][dim_row] (each column-major), V[0] holding timeslice v_t0 (0: all Lt
// resident; a ring slot otherwise).  vdv: [2*n_ops][Lt][nev][nev].
constexpr int kVdvFp64Ops = 3;
cudaError_t vdaggerv_fp64(double2 *vdv, double2 const *V, VdvFamily const *fam, int32_t n_fam,
                          int32_t t0, int32_t nt, Geometry g, cudaStream_t stream,
                          int32_t v_t0 = 0);
// Split-BF16 tensor-core VdaggerV (vdv_tc.cu): same result as vdaggerv_fp64
// to ~1e-13 relative.  The plan of an operator table: families (planes of
// constant x, or the whole lattice where those are too small) of the momentum
// operators, then one family per displaced operator; all pointers are device
// memory kept by the caller.
// Columns of B.  The rows of an M tile are 64 eigenvectors; where the last tile
// would hold few, its rows i >= full of the phase families come from edge columns
// instead: sum_x V_i conj(phase) conj(V_j) is conj(G(i, j)), with V_i as a column and
// the rows j < full.  Order: (f, j < full) family by family, (f, j >= full), then the
// edge columns (f, i) of the families n_lead <= f < n_mom (those before are
// Hermitian).  full = nev: no edge columns, the plain order f nev + j.
struct VdvColumns {
  int32_t nev, n_fam, n_mom, n_lead, full;
  __host__ __device__ int64_t n_cols() const { return static_cast<int64_t>(n_fam) * nev; }
  __host__ __device__ int64_t n_all() const {
    return n_cols() + static_cast<int64_t>(n_mom - n_lead) * (nev - full);
  }
  __host__ __device__ int64_t pos(int32_t f, int32_t j) const {
    return j < full ? static_cast<int64_t>(f) * full + j
                    : static_cast<int64_t>(n_fam) * full +
                          static_cast<int64_t>(f) * (nev - full) + (j - full);
  }
  __host__ __device__ int64_t edge(int32_t f, int32_t i) const {
    return n_cols() + static_cast<int64_t>(f - n_lead) * (nev - full) + (i - full);
  }
  __host__ __device__ bool phase(int32_t f) const { return f >= n_lead && f < n_mom; }
  // Column c < n_all(): family and eigenvector; true for an edge column.
  __host__ __device__ bool decode(int64_t c, int32_t &f, int32_t &j) const {
    int64_t const inner = static_cast<int64_t>(n_fam) * full;
    if (c < inner) {
      f = static_cast<int32_t>(c / full);
      j = static_cast<int32_t>(c % full);
      return false;
    }
    bool const e = c >= n_cols();
    int64_t const q = c - (e ? n_cols() : inner);
    f = static_cast<int32_t>(q / (nev - full)) + (e ? n_lead : 0);
    j = static_cast<int32_t>(q % (nev - full)) + full;
    return e;
  }
};
struct VdvTcPlan {
  int32_t n_fam, n_mom;           // families; those of momentum operators come first
  VdvColumns cols;
  int32_t n_planes, per;          // planes, lattice entries (3 x sites) of each
  VdvFamily const *fam;           // [n_fam]
  longlong2 const *phase_fx;      // [n_fam][per / 3]: the families' phases x 2^62
  double2 const *roots;           // [n_planes]: e^{-2 pi i n / n_planes}
  int2 const *mn;                 // GEMM tiles (m, n) of one plane
  int32_t n_mn;
};
// The columns and (m, n) tiles of one plane, without the tiles of which no entry is
// wanted (below the diagonal of Hermitian families; the last M tile where edge
// columns stand in for it).  Edge columns are taken where they cost less.
std::vector<int2> vdaggerv_tc_tiles(std::vector<VdvFamily> const &fam, int32_t n_mom,
                                    int32_t nev, int32_t n_planes, int32_t sm_count,
                                    VdvColumns &cols);
// Scratch for `batch` timeslices per GEMM launch.
size_t vdaggerv_tc_scratch_bytes(Geometry g, VdvTcPlan const &pl, int32_t batch);
// phase_fx[k] = round(phase[k] 2^62) per component, the fixed-point phases the
// split-precision VdaggerV multiplies with integer arithmetic.
cudaError_t phase_fixed(longlong2 *phase_fx, double2 const *phase, int64_t n,
                        cudaStream_t stream);
// roots[n] = e^{-2 pi i n / n_planes}.
cudaError_t unit_roots(double2 *roots, int32_t n_planes, cudaStream_t stream);
// Timeslices per GEMM launch for n_t timeslices: at most what max_bytes of
// scratch holds; the fewest whose rounds of one tile per SM, over all
// launches, are within 2% of the least.
int32_t vdaggerv_tc_batch(Geometry g, VdvTcPlan const &pl, int32_t sm_count, size_t max_bytes,
                          int32_t n_t);
// Displaced operators of the split-precision VdaggerV: family n_mom + d is
// V_t^H D_d(V_t), D_d the displacement steps of operator d (displaced_vectors
// above), momentum not applied.
constexpr int kMaxDispSteps = 8;
struct VdvDisplaced {
  int32_t n;                     // number of displaced operators
  int32_t const *n_steps;        // host: steps per operator
  int32_t const *steps;          // host: [n][kMaxDispSteps][2] (dir 0..2, forward 0/1)
  double2 const *U;              // device: links [Lt][site][dir][9]
  double2 const *P;              // device: line_products of U, null without backward steps
  double2 *W;                    // device scratch of displaced_vectors
};
cudaError_t vdaggerv_tc(double2 *vdv, double2 const *V, VdvTcPlan const &pl, int32_t t0,
                        int32_t nt, Geometry g, void *scratch, size_t scratch_bytes, int *err,
                        cudaStream_t stream, cudaEvent_t const *t_ready = nullptr,
                        VdvDisplaced const *disp = nullptr,
                        cudaEvent_t const *gemm_ev = nullptr, int32_t n_gemm_ev = 0,
                        int32_t v_t0 = 0);
// (V: consecutive timeslices, V[0] holding timeslice v_t0.  scratch: at least
// vdaggerv_tc_scratch_bytes of one timeslice; err: device int, set non-zero
// when a bounded wait gave up.  t_ready[t], when given and non-null: event
// after which timeslice t of V is valid; the slicing of t waits for it on
// `stream`.  gemm_ev: when given, the events 2k and 2k+1 are recorded on
// `stream` just before and after the k-th GEMM launch, for k < n_gemm_ev / 2;
// vdaggerv_tc_gemm_launches gives k's range.)
int32_t vdaggerv_tc_gemm_launches(int32_t nt, int32_t batch);
// One bounded mbarrier wait that nothing completes (selftest.cu): *err = 1
// once it gives up after `cycles` clock cycles.
cudaError_t bounded_wait_selftest(int *err, long long cycles, cudaStream_t stream);
// Identity blocks for code 2*op (and 2*op+1).
cudaError_t vdaggerv_identity(double2 *vdv, int32_t op, Geometry g, cudaStream_t stream);
// vdv[2*op+1][t] = vdv[2*op][t]^H for all ops, t.
cudaError_t vdaggerv_daggers(double2 *vdv, int32_t n_ops, Geometry g, cudaStream_t stream);

// Factor intermediates and factors (src/DilutedFactorFactory.cpp:34-253).
cudaError_t q0m(double2 *out, Q0MInst const *inst, int64_t n, double2 const *vdv,
                double2 const *noise, Geometry g, cudaStream_t stream);
cudaError_t q1r(double2 *out, Q1RInst const *inst, int64_t n, double2 const *vdv,
                double2 const *noise, Geometry g, cudaStream_t stream);
cudaError_t q2m(double2 *out, Q2MInst const *inst, int64_t n, double2 const *vdv,
                double2 const *peram, Geometry g, cudaStream_t stream);
cudaError_t q0(double2 *slots, Q0Inst const *inst, int64_t n, double2 const *q0m,
               double2 const *noise, Geometry g, cudaStream_t stream);
cudaError_t q1(double2 *slots, Q1Inst const *inst, int64_t n, double2 const *q1r,
               double2 const *peram, Geometry g, cudaStream_t stream);
cudaError_t q2(double2 *slots, Q2Inst const *inst, int64_t n, double2 const *q2m,
               double2 const *peram, Geometry g, cudaStream_t stream);
// Q1 factors that share their products: x is scratch of n_x 64 dilE^2 entries.
cudaError_t q1_shared(double2 *slots, double2 *x, X1Inst const *xi, int64_t n_x,
                      Q1Pick const *picks, int64_t n, double2 const *q1r, double2 const *peram,
                      Geometry g, cudaStream_t stream);

// slots[c] = slots[a] * slots[b] (operator*, src/DilutedFactor.cpp:6-51).
cudaError_t products(double2 *slots, ProdInst const *p, int64_t n, int32_t eds,
                     cudaStream_t stream);

// Trace values of every entry of the lists lists[which[0..n_which)]
// (factor_to_trace, src/DilutedTrace.cpp:84-165), entry e of list L at
// values[L.val_off + e * L.stride].  shape_i/shape_j: entry operand indices,
// shape_off: [n_shapes+1] offsets into them.
cudaError_t traces(double2 *values, TraceList const *lists, int32_t const *which,
                   int64_t n_which, int32_t const *shape_i, int32_t const *shape_j,
                   int64_t const *shape_off, double2 const *slots, int32_t eds,
                   cudaStream_t stream);

// Mixed path: matrices in double-float form (float4 = re hi, re lo, im hi, im lo
// per complex), as stored and transposed; traces as compensated FP32 dot products
// over unit-stride operands.
// Mixed path: FP64 -> double-float (float4) copy.
cudaError_t to_df(float4 *dst, double2 const *src, int64_t n, cudaStream_t stream);
// Mixed path: the Q0M and Q1R intermediates and the Q0 factors in double-float;
// Q0 written into the slot buffers in both layouts (sn stored, st transposed),
// the largest |re|, |im| of their slots (slot_maxbits) added to slot_bits.
cudaError_t factors_df(float4 *sn, float4 *st, float4 *q0m_buf, float4 *q1r_buf,
                       Q0MInst const *q0m_i, int64_t n_q0m, Q1RInst const *q1r_i, int64_t n_q1r,
                       Q0Inst const *q0_i, int64_t n_q0, float4 const *vdv, float4 const *noise,
                       unsigned int *slot_bits, Geometry g, cudaStream_t stream);
// slots[c] = slots[a] * slots[b] in double-float, both layouts written.
cudaError_t products_df(float4 *slots_n, float4 *slots_t, ProdInst const *p, int64_t n,
                        int32_t eds, cudaStream_t stream);
// The same products on the tensor cores (product_tc.cu), for eds = 8 .. 32 and 64.
// Matrices are padded to P = prod_tc_pad(eds) rows and columns in the operands
// (not in the slots).  The products of one dependency level come in groups of up
// to 64 / P left matrices (slots l[0..n_l)) with the union of their right matrices:
// column block u of group g is right matrix u_list[g.u_off + u] (an index into
// the level's r_slots) and out_tab[4 (g.u_off + u) + l] is four times the slot of
// product l x u plus the layouts in which it is read (1 natural, 2 transposed; for
// eds = 64 both are written all the same), or -1 when the level does not ask for
// it.  Tiles: (group, n tile of
// 80 columns).  Scratch: the groups' A regions (prod_tc_a_bytes each) from 0,
// the right-matrix streams (prod_tc_r_bytes each) from r_off; exponents: 64
// per group from 0, eds per right matrix from r_expo.  slot_bits (as
// slot_maxbits; zero for the level's product slots before the call) receives
// the largest |re|, |im| of every product written.
struct ProdGroup {
  int32_t l[4];   // left-matrix slots
  int32_t n_l;    // left matrices in the group (1 .. 64 / eds)
  int32_t n_u;    // right matrices in the union
  int32_t u_off;  // first column block in u_list / out_tab
  int32_t ea;     // exponent index of the group's row 0 (64 g)
};
// One unit of GEMM work.  eds = 64: the 80-column tile nt of the group.  eds <= 32:
// the n (at most kProdSteps) right matrices u_list[u .. u + n) of the group, one
// GEMM step each; n_l and ea repeat the group's.
constexpr int32_t kProdSteps = 32;
struct ProdTile {
  int32_t group, nt;
  int32_t u, n, n_l, ea;
};
// (4 x 4 matrices fill 1/16 of a padded product and stay with the double-float
// kernel, as those between 32 and 64 do, whose left operand leaves no room for
// the right ones.)
inline bool prod_tc_steps(int32_t eds) { return eds >= 8 && eds <= 32; }
inline bool prod_tc_supported(int32_t eds) { return prod_tc_steps(eds) || eds == 64; }
__host__ __device__ inline int32_t prod_tc_pad(int32_t eds) {
  return eds <= 16 ? 16 : eds <= 32 ? 32 : 64;
}
__host__ __device__ inline int64_t prod_tc_r_bytes(int32_t eds) {
  // (P / 16) k-tiles x 6 slices x P columns x 64 bytes
  return 24LL * prod_tc_pad(eds) * prod_tc_pad(eds);
}
int64_t prod_tc_a_bytes(int32_t eds);
cudaError_t products_tc(float4 *slots_n, float4 *slots_t, uint8_t *scratch, int64_t r_off,
                        int32_t *expo, int64_t r_expo, ProdGroup const *groups, int64_t n_groups,
                        int32_t const *r_slots, int64_t n_r, int32_t const *u_list,
                        int32_t const *out_tab, ProdTile const *tiles, int64_t n_tiles,
                        int32_t eds, unsigned int *slot_bits, int *err, cudaStream_t stream);
// Trace values (FP64 sums of the double-float results), laid out as for traces().
cudaError_t traces_df(double2 *values, TraceList const *lists, int32_t const *which,
                      int64_t n_which, int32_t const *shape_i, int32_t const *shape_j,
                      int64_t const *shape_off, float4 const *slots_n, float4 const *slots_t,
                      int32_t eds, cudaStream_t stream);
// Dense trace groups on the tensor cores (trace_tc.cu).  One matrix slot
// sliced into the operand stream of a GEMM region:
struct TrSlice {
  int64_t dst;   // byte offset of the region in the scratch buffer
  int32_t slot;  // matrix slot
  int32_t row;   // complex row (A region) or column (B region) of the matrix
  int32_t expo;  // index of the matrix's exponent in the exponent array
  int32_t pad;
};
// Matrices of one 8-row core-matrix group of a region, sliced together so that
// every store covers whole core matrices: kTrSliceRowsA consecutive complex
// rows of an A region (eight rows of A', two per matrix) or kTrSliceRowsB
// consecutive columns of a B region, from a row that is a multiple of that
// count; exponent indices expo0, expo0 + 1, ...
constexpr int32_t kTrSliceRowsA = 4, kTrSliceRowsB = 8;
struct TrSliceGroup {
  int64_t dst;    // byte offset of the region in the scratch buffer
  int32_t row0;   // first row (A) or column (B) of the group
  int32_t n;      // matrices in the group (1 .. 4 for A, 1 .. 8 for B)
  int32_t expo0;  // exponent index of the first matrix
  int32_t slot[8];
  int32_t pad;
};
// One output tile of 64 rows x 80 columns of one GEMM.  tab < 0: value (r, c) at
// out + c ld + r (kTabRelative, tc_gemm_df only: without the factor 2^e of its row's
// exponent e).  Otherwise the rows are stacked blocks of n_a operand groups
// and the columns of n_b: row r of the tile is group ia of block u, (row0 + r) =
// u n_a + ia, column c group ib of block v, (col0 + c) = v n_b + ib, and the
// value belongs to entry e = entries[tab + u tab_ld + v] (none when negative),
// at out + e n_a n_b + ib n_a + ia.
struct TrTile {
  int64_t a_src, b_src;  // byte offsets of the tile's A and B operand streams
  int64_t out;           // value index (see above)
  int64_t tab;
  int32_t ea, eb;        // exponent indices of tile row 0 and column 0
  int32_t rows, cols;    // valid rows (<= 64) and columns (<= 80)
  int32_t ld;            // tab < 0: value index distance between columns
  int32_t n_a, n_b, row0, col0, tab_ld;
};
constexpr int32_t kTrTileRows = 64, kTrTileCols = 80;
constexpr int64_t kTabRelative = -2;
constexpr int32_t kTrGroupBits = 16;  // v << kTrGroupBits | ib in the epilogue: n_b <= 2^16
int64_t trace_tc_k_tiles(int32_t eds);
size_t trace_tc_a_bytes(int32_t rows, int32_t eds);  // A region of `rows` matrices
size_t trace_tc_b_bytes(int32_t cols, int32_t eds);  // B region of `cols` matrices
// Largest |re|, |im| of each matrix slot first..first+n (double-float,
// natural layout, high words) as float bits: the slicing of the trace
// operands takes each matrix's exponent from it instead of scanning the
// matrix again for each group region it appears in.
cudaError_t slot_maxbits(unsigned int *bits, float4 const *slots, int64_t first, int64_t n,
                         int32_t eds, cudaStream_t stream);
// Slices the A matrices (natural layout, conjugated) and B matrices
// (transposed layout) of a batch into their regions of `scratch`, one row
// group per CTA, with the largest entries of their slots (slot_maxbits).
cudaError_t trace_tc_slice(uint8_t *scratch, int32_t *expo, TrSliceGroup const *a_groups,
                           int64_t n_a, TrSliceGroup const *b_groups, int64_t n_b,
                           float4 const *slots_n, float4 const *slots_t,
                           unsigned int const *slot_bits, int32_t eds, cudaStream_t stream);
// The GEMM tiles of a batch; FP64 trace values into `values`.
cudaError_t trace_tc_gemm(double2 *values, uint8_t const *scratch, int32_t const *expo,
                          TrTile const *tiles, int64_t n_tiles, int32_t const *entries,
                          int32_t eds, int *err, cudaStream_t stream);

// Generic form of the same GEMM (factor_tc.cu): k_tiles k-tiles of 16
// complex entries; region sizes for `rows` A rows / `cols` B columns.
size_t tc_a_bytes(int32_t rows, int32_t k_tiles);
size_t tc_b_bytes(int32_t cols, int32_t k_tiles);
int32_t gemm_k_tiles(int64_t K);
cudaError_t tc_gemm(double2 *out, uint8_t const *scratch, int32_t const *expo,
                    TrTile const *tiles, int64_t n_tiles, int32_t k_tiles, int *err,
                    cudaStream_t stream, int32_t const *entries = nullptr);
// The same with double-float results (re_hi, re_lo, im_hi, im_lo), for plain
// tiles: the short K of the factor GEMMs leaves no time for FP64 conversions.
cudaError_t tc_gemm_df(float4 *out, uint8_t const *scratch, int32_t const *expo,
                       TrTile const *tiles, int64_t n_tiles, int32_t k_tiles, int *err,
                       cudaStream_t stream);

// One GEMM operand row (A) or column (B) gathered from up to four strided
// segments of a source array, each with an exact factor (0: +1, 1: +i, 2: -1,
// 3: -i).  K = n_seg * seg_len, zero-padded to the region's k-tiles.  In a relative
// source (kTabRelative) a segment is without the factor 2^e of the exponent at e_row.
struct GSeg {
  int64_t src;
  int32_t factor;
  int32_t e_row;
};
constexpr int kGMaxSeg = 4;
struct GVec {
  int64_t dst;     // byte offset of the region in the scratch buffer
  int64_t stride;  // element stride along K inside a segment
  int32_t row;     // row (A) or column (B) within the region
  int32_t expo;    // index of its exponent
  int32_t n_seg, seg_len;
  int32_t pad[2];  // to 26 words: eight in shared memory, the same word of each, meet no bank twice
  GSeg seg[kGMaxSeg];
};
// Up to eight consecutive operand vectors of one region, items[first .. first +
// n), the first one's row a multiple of 8.
struct GVecGroup {
  int64_t first;
  int32_t n, pad;
};
// Slices the operand vectors of n groups (A rows with put conj(v) when conj, or B
// columns) from an FP64, a double-float or a relative double-float source.
cudaError_t gvec_slice_f64(uint8_t *scratch, int32_t *expo, GVecGroup const *groups, int64_t n,
                           GVec const *items, bool is_a, bool conj, double2 const *src, int32_t k_tiles,
                           cudaStream_t stream);
cudaError_t gvec_slice_df(uint8_t *scratch, int32_t *expo, GVecGroup const *groups, int64_t n,
                          GVec const *items, bool is_a, bool conj, float4 const *src, int32_t k_tiles,
                          cudaStream_t stream);
cudaError_t gvec_slice_relative(uint8_t *scratch, int32_t *expo, GVecGroup const *groups,
                                int64_t n, GVec const *items, float4 const *src, int32_t k_tiles,
                                cudaStream_t stream);  // A rows, conjugated
// Q1 factor slots from the dense product X1 (factor_tc.cu); Q2 slots from the
// dense Q2 GEMM output; both double-float, as tc_gemm_df writes them.  need: the
// layouts to write (1 stored, 2 transposed); slot_bits: largest |re|, |im| of
// the slot (slot_maxbits).
struct Q1Gather {
  int64_t x_off;  // element offset of X1 of the factor's timeslice
  int32_t ld, row0, col0, gamma, slot, need;
};
struct Q2Gather {
  int64_t off;  // element offset of the factor's (0, 0) entry
  int32_t ld, slot, need, pad;
};
cudaError_t upload_gamma_tc(cudaStream_t stream);
cudaError_t q1_gather(float4 *sn, float4 *st, unsigned int *slot_bits, Q1Gather const *g,
                      int64_t n, float4 const *x, int32_t dilE, cudaStream_t stream);
cudaError_t q2_gather(float4 *sn, float4 *st, unsigned int *slot_bits, Q2Gather const *g,
                      int64_t n, float4 const *y, int32_t eds, cudaStream_t stream);

// Term values (resolve_request / inner_product, src/Diagram.cpp:9-94,
// src/DilutedTrace.cpp:5-82) with the native (0) or Kahan (1) accumulator.
cudaError_t terms(double2 *term_val, Term const *t, int64_t n, TraceList const *lists,
                  double2 const *values, uint16_t const *shape_mask,
                  int64_t const *shape_off, int32_t kahan, cudaStream_t stream);

// running[o] += term_val[idx[k]] for k in [seg[o], seg[o+1]) in order
// (Diagram::assemble, src/Diagram.cpp:96-114).
cudaError_t accumulate(double2 *running, int32_t const *seg_out, int64_t const *seg_off,
                       int64_t n_seg, int32_t const *idx, double2 const *term_val,
                       cudaStream_t stream);
// x[k] /= d for k < n (both components).
cudaError_t divide(double2 *x, int64_t n, double d, cudaStream_t stream);

}  // namespace dev
}  // namespace slaph
