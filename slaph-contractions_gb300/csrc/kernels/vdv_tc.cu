// Split-BF16 tensor-core VdaggerV (tcgen05, sm_103a).
//
// VdaggerV = V^H diag(phase) V (src/OperatorFactory.cpp:292-300) with FP64
// inputs and an FP64-accurate result from BF16 tensor-core products, by the
// split-BF16 scheme of tc_common.cuh: A' rows are the eigenvectors V_i, B
// columns W_j = diag(phase) V_j, K' = 2 * 3L^2 per plane; rows are scaled by the
// exponent of the eigenvector's largest |entry| (the same for W, |phase| = 1).
//
// Operators come in momentum families (vdv_families.hpp): the GEMM gives the
// sums over planes of constant x, one set of B columns per family, and
// vdv_fourier_kernel the operators from them, so that operators that differ in
// p_x only share their GEMM work, and tiles below the diagonal of a Hermitian
// family are not computed.  16 operators with |p|^2 <= 4 are 7 families, 13
// with |p|^2 <= 3 are 5, 3 with |p|^2 <= 1 are 3.  The planes are also what
// fills the chip: a timeslice gives n_planes times as many tiles as a sum over
// the whole lattice, so a launch needs few timeslices (and little scratch) for
// an even load.  (Slicing the next timeslices on a second stream during a GEMM
// gains nothing but the last round: the GEMM's ten warps of 168 registers leave
// no room for another CTA on an SM.)
//
// Data path: V is read once per timeslice to write the A slices and the B
// slices of all families to HBM, already in the tcgen05 core-matrix layout,
// from where the GEMM streams them into shared memory.  The B columns of all
// families form one N dimension (column f nev + j: family f, eigenvector j),
// cut into tiles of kTN without padding between families.  Padding rows and
// columns of the last tiles are not written: they only reach output rows and
// columns that nobody reads.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.cuh"
#include "norm_max.cuh"
#include "tc_common.cuh"

namespace slaph {
namespace dev {

namespace {

using namespace tc;

// K tiles (kTK / 2 complex entries) of one plane; planes are padded to whole
// K tiles.
__host__ __device__ inline int32_t plane_k_tiles(int32_t per) {
  return (per + kTK / 2 - 1) / (kTK / 2);
}

// Exponent e with sqrt(n2) (1 + 1e-15) < 2^e, 0 for n2 = 0.
__device__ __forceinline__ int expo_of_norm2(double n2) {
  int e = 0;
  double const m = sqrt(n2);
  if (m > 0) frexp(m * (1.0 + 1e-15), &e);
  return e;
}

// norms[slot][i] of columns i of V, timeslice blockIdx.z (slots at slot_bytes),
// one warp per kNormChunk entries: 5.5 TB/s, against 2.5 TB/s for FP64 norms.
constexpr int kNormChunk = 2048;  // entries per warp
__global__ void __launch_bounds__(32)
    norm_kernel(uint8_t *norms, size_t slot_bytes, double2 const *V, Geometry g) {
  int const i = blockIdx.y;
  double2 const *col = V + (static_cast<int64_t>(blockIdx.z) * g.nev + i) * g.dim_row;
  int64_t const b = static_cast<int64_t>(blockIdx.x) * kNormChunk;
  int64_t const e = min(g.dim_row, b + kNormChunk);
  NormMax m{0, 0};
#pragma unroll 8
  for (int64_t x = b + threadIdx.x; x < e; x += 32) norm_max(m, col[x]);
  norm_max_add(reinterpret_cast<NormMax *>(norms + blockIdx.z * slot_bytes) + i, m);
}

// Exponents e_i with max_x |V(x, i)| < 2^e_i from the columns' norms, one warp
// per column; where the norm does not settle the exponent the column is read
// again in FP64.  The norms are zeroed for their next use.
__global__ void __launch_bounds__(32)
    expo_kernel(uint8_t *norms, uint8_t *expo, size_t slot_bytes, double2 const *V, Geometry g) {
  int const i = blockIdx.x, lane = threadIdx.x;
  NormMax *m = reinterpret_cast<NormMax *>(norms + blockIdx.y * slot_bytes) + i;
  NormMax const x = *m;
  double const n = static_cast<double>(__uint_as_float(x.n2));
  int ex = expo_of_norm2(n * (1.0 - 0x1p-20));
  // within 2^-50 .. 2^50 the squares stay in the FP32 range
  bool const fits = x.top >= (973u << 20) && x.top < (1073u << 20);
  if (!fits || ex != expo_of_norm2(n * (1.0 + 0x1p-20))) {
    double2 const *col = V + (static_cast<int64_t>(blockIdx.y) * g.nev + i) * g.dim_row;
    double mx = 0;
#pragma unroll 4
    for (int64_t k = lane; k < g.dim_row; k += 32) {
      double2 const v = col[k];
      mx = fmax(mx, v.x * v.x + v.y * v.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    ex = expo_of_norm2(mx);
  }
  __syncwarp();
  if (lane == 0) {
    reinterpret_cast<int32_t *>(expo + blockIdx.y * slot_bytes)[i] = ex;
    *m = NormMax{0, 0};
  }
}

// Slices of timeslice blockIdx.y (slots at slot_bytes).  kA: the A slices of V, [m_tile][K tile][slice][kTM x
// kTK]; kB: the B slices of phase_f V for the families f0 .. f0 + n_fam - 1 at their
// columns (VdvColumns), [n_tile][K tile][slice][kTN x kTK]; kEdge: their edge columns,
// of the eigenvectors from cols.full on with the conjugate phase (a launch of its own:
// as a second pass of the loop over families it slowed every launch by a tenth).
//
// A warp covers eight eigenvectors in one K tile: lane (r, kg) = (lane % 8,
// lane / 8) takes eigenvector 8 rg + r and the 4 complex K entries 4 kg .. 4 kg
// + 3 of the tile, i.e. one 16-byte row of a core matrix.  V is read and put in
// fixed point once for all of it; the phase product is taken in fixed point
// with integer operations only: with V = F_v 2^(e-55) and phase = P 2^-62
// (|P| <= 2^62), W = ((F_v 4) P / 2^64) 2^(e-55), the high word of a 128-bit
// product.  The A rows of an eigenvector are a row pair (Re v, Im v) and (-Im v,
// Re v): a lane fetches the packed words of the eigenvector whose row it stores
// by warp shuffles (the second row is the first with its halves swapped and one
// sign flipped), so that every slice store of a warp, A or B, fills whole
// 128-byte core matrices (512 contiguous bytes).  Bound by HBM: 16 bytes read,
// 48 (A) and 24 per family (B) written per entry.  With A, four CTAs per SM (64
// registers instead of 80) run at 5.9 TB/s, three at 5.6 (32^3x64 Nev 220: 31.6 ms
// and 33.2).
template <bool kA, bool kB, bool kEdge>
__global__ void __launch_bounds__(256, kA ? 4 : 1)
    slice_kernel(uint8_t *a_out, uint8_t *b_out, size_t slot_bytes, double2 const *V,
                 longlong2 const *phase_fx, int32_t n_fam, uint8_t const *expos, int32_t n_planes,
                 int32_t per, VdvColumns cols, int32_t f0, Geometry g) {
  a_out += blockIdx.y * slot_bytes;
  b_out += blockIdx.y * slot_bytes;
  int32_t const *expo = reinterpret_cast<int32_t const *>(expos + blockIdx.y * slot_bytes);
  double2 const *Vt = V + static_cast<int64_t>(blockIdx.y) * g.nev * g.dim_row;
  int64_t const wid = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) / 32;
  int const lane = threadIdx.x % 32;
  int32_t const ktp = plane_k_tiles(per);
  int64_t const k_tiles = static_cast<int64_t>(ktp) * n_planes;
  int const first = kEdge ? cols.full / 8 : 0;  // group of eight eigenvectors
  int64_t const groups = (g.nev + 7) / 8 - first;
  if (wid >= groups * k_tiles) return;
  int64_t const kt = wid / groups;
  int const rg = first + static_cast<int>(wid % groups);
  int const r = lane % 8, kg = lane / 8;
  int const j = rg * 8 + r;
  bool const row_ok = j < g.nev;
  int32_t const plane = static_cast<int32_t>(kt / ktp);
  int32_t const k0 = static_cast<int32_t>(kt - static_cast<int64_t>(plane) * ktp) * (kTK / 2) +
                     4 * kg;  // first entry within the plane
  long long vr[4], vi[4];
  int32_t site[4];
  int const e = row_ok ? expo[j] : 0;
  double2 const *src = Vt + static_cast<int64_t>(j) * g.dim_row + static_cast<int64_t>(plane) * per;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    int32_t const k = k0 + q;
    bool const in = row_ok && k < per;
    double2 const v = in ? src[k] : make_double2(0, 0);
    vr[q] = fixed55(v.x, e);
    vi[q] = fixed55(v.y, e);
    site[q] = in ? k / 3 : 0;
  }
  if (kA) {
    uint32_t w[kSlices][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float dre[kSlices], dim[kSlices];
      digits6(vr[q], dre);
      digits6(vi[q], dim);
#pragma unroll
      for (int s = 0; s < kSlices; ++s) w[s][q] = bf16x2(dre[s], dim[s]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // the two core-matrix groups of the 16 A rows
      int const from = 4 * h + r / 2 + 8 * kg;
      int const i = rg * 8 + 4 * h + r / 2;
      int const arow = 2 * (i % (kTM / 2)) + (r & 1);
      uint8_t *dst = a_out + (static_cast<int64_t>(i / (kTM / 2)) * k_tiles + kt) * kStageA +
                     ((arow >> 3) * 4 + kg) * 128 + (arow & 7) * 16;
#pragma unroll
      for (int s = 0; s < kSlices; ++s) {
        uint32_t x[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t const y = __shfl_sync(0xffffffffu, w[s][q], from);
          x[q] = (r & 1) ? __byte_perm(y, 0, 0x1032) ^ 0x8000u : y;
        }
        if (i < g.nev)
          *reinterpret_cast<uint4 *>(dst + s * kABlk) = make_uint4(x[0], x[1], x[2], x[3]);
      }
    }
  }
  if (kB && row_ok) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      vr[q] *= 4;
      vi[q] *= 4;
    }
    int32_t const sites = per / 3;
    // columns of eigenvector j, family after family (below 2^31)
    uint32_t gc = static_cast<uint32_t>(kEdge ? cols.edge(f0, j) : cols.pos(f0, j));
    uint32_t const gstep = kEdge || j >= cols.full ? g.nev - cols.full : cols.full;
    for (int f = 0; f < n_fam; ++f, gc += gstep) {
      longlong2 const *ph = phase_fx + static_cast<int64_t>(f) * sites;
      uint32_t w[kSlices][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        longlong2 p = ph[site[q]];
        if (kEdge) p.y = -p.y;
        long long const wr = __mul64hi(vr[q], p.x) - __mul64hi(vi[q], p.y);
        long long const wi = __mul64hi(vr[q], p.y) + __mul64hi(vi[q], p.x);
        float dre[kSlices], dim[kSlices];
        digits6(wr, dre);
        digits6(wi, dim);
#pragma unroll
        for (int s = 0; s < kSlices; ++s) w[s][q] = bf16x2(dre[s], dim[s]);
      }
      int64_t const nt = gc / kTN;
      int const rr = static_cast<int>(gc % kTN);
      uint8_t *dst =
          b_out + (nt * k_tiles + kt) * kStageB + ((rr >> 3) * 4 + kg) * 128 + (rr & 7) * 16;
#pragma unroll
      for (int s = 0; s < kSlices; ++s)
        *reinterpret_cast<uint4 *>(dst + s * kBBlk) =
            make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
    }
  }
}

__global__ void phase_fixed_kernel(longlong2 *dst, double2 const *src, int64_t n) {
  int64_t const k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (k >= n) return;
  double2 const v = src[k];
  dst[k] = make_longlong2(__double2ll_rn(ldexp(v.x, 62)), __double2ll_rn(ldexp(v.y, 62)));
}

__global__ void unit_roots_kernel(double2 *roots, int32_t n) {
  int32_t const k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double s, c;
  sincospi(2.0 * static_cast<double>(k) / static_cast<double>(n), &s, &c);
  roots[k] = make_double2(c, -s);
}

// Tile i of a launch: (m, n) tile mn[i % n_mn] of plane (i / n_mn) % n_planes
// of batch slot i / (n_mn n_planes) (timeslice t0 + slot).  Slot b has its own A
// slices, B slices, plane sums and exponents at stride slot_bytes in the
// scratch buffer: the eigenvectors' exponents, then per family f >= n_mom
// (displaced) the exponents of its B columns at (1 + f) nev.
struct VdvTiles {
  uint8_t const *scratch;
  size_t slot_bytes, b_off, e_off;
  int2 const *mn;
  int32_t n_mn, n_planes, k_tiles;  // k_tiles: of one plane
  __device__ __forceinline__ void decode(int i, int &mt, int &nt, int &plane, int &slot) const {
    int2 const t = mn[i % n_mn];
    mt = t.x;
    nt = t.y;
    plane = (i / n_mn) % n_planes;
    slot = i / (n_mn * n_planes);
  }
  struct Ctx {
    uint8_t const *a, *b;
  };
  __device__ __forceinline__ Ctx context(int i, int lane) const {
    int mt, nt, plane, slot;
    decode(i, mt, nt, plane, slot);
    uint8_t const *sbase = scratch + slot * slot_bytes;
    int64_t const at = static_cast<int64_t>(plane) * k_tiles;
    int64_t const all = static_cast<int64_t>(n_planes) * k_tiles;
    return Ctx{sbase + (mt * all + at) * kStageA, sbase + b_off + (nt * all + at) * kStageB};
  }
  __device__ __forceinline__ void load(Ctx const &c, int kt, uint8_t *dst, uint64_t *bar,
                                       int lane) const {
    if (lane == 0) load_contiguous(c.a, c.b, kt, dst, bar, 0);
  }
};

// Epilogue of one tile: D = (hi + lo) 2^(e_i + f_c - 14), rows (2i, 2i+1) =
// (Re, Im) of the plane sum G(i, j) of family f for the tile's B columns c = (f, j),
// written to sums[((plane n_fam + f) nev + j) nev + i] of the slot, of an edge column
// (f, k) conjugated to entry (k, i); e: exponents of the eigenvectors (A rows), f:
// those of the B columns (the eigenvectors' for momentum families, |phase| = 1; those
// of D(V) for the displaced ones, f >= n_mom, at (1 + f) nev).  A warp stores 16
// consecutive i of a column: 256 bytes.
struct VdvEpilogue {
  VdvTiles tl;
  size_t s_off;
  VdvColumns cols;
  struct Pre {};
  __device__ __forceinline__ Pre prepare(int, int, int) const { return Pre{}; }
  __device__ __forceinline__ void operator()(Pre const &, int it, int row, int col0,
                                             float const (&hi)[kColsW],
                                             float const (&lo)[kColsW]) const {
    int mt, nt, plane, slot;
    tl.decode(it, mt, nt, plane, slot);
    int const nev = cols.nev, lane = threadIdx.x % 32;
    int const i = mt * (kTM / 2) + row / 2;
    uint8_t const *sbase = tl.scratch + slot * tl.slot_bytes;
    int32_t const *expo = reinterpret_cast<int32_t const *>(sbase + tl.e_off);
    double *sums = reinterpret_cast<double *>(const_cast<uint8_t *>(sbase) + s_off) +
                   2 * static_cast<int64_t>(plane) * cols.n_cols() * nev + (row & 1);
    int const ei = i < nev ? expo[i] : 0;
    // Lane k looks up the warp's columns k and 32 + k; the column loop takes them by
    // warp shuffles.  at: offset of the entry for i = 0; kind: 1 wanted, 2 edge, 4 only
    // for i < full (what edge columns, or the columns they stand in for, hold beyond
    // belongs to other columns).
    int64_t at[2];
    int ex[2], kind[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int64_t const c = static_cast<int64_t>(nt) * kTN + col0 + 32 * h + lane;
      at[h] = 0;
      ex[h] = kind[h] = 0;
      if (32 * h + lane >= kColsW || c >= cols.n_all()) continue;
      int32_t f, j;
      bool const edge = cols.decode(c, f, j);
      at[h] = (static_cast<int64_t>(f) * nev + (edge ? 0 : j)) * nev + (edge ? j : 0);
      ex[h] = f < cols.n_mom ? expo[j] : expo[(1 + f) * nev + j];
      kind[h] = 1 | (edge ? 2 : 0) | (edge || (j < cols.full && cols.phase(f)) ? 4 : 0);
    }
#pragma unroll
    for (int c = 0; c < kColsW; ++c) {
      int const ec = __shfl_sync(0xffffffffu, ex[c / 32], c % 32);
      int const kd = __shfl_sync(0xffffffffu, kind[c / 32], c % 32);
      int64_t const a = __shfl_sync(0xffffffffu, at[c / 32], c % 32);
      if (!(kd & 1) || i >= ((kd & 4) ? cols.full : nev)) continue;
      double const v = df_scaled(hi[c], lo[c], ei + ec - 14);
      if (kd & 2)
        sums[2 * (a + static_cast<int64_t>(i) * nev)] = (row & 1) ? -v : v;
      else
        sums[2 * (a + i)] = v;
    }
  }
};

// The GEMM: n_mn x n_planes x batch tiles over persistent CTAs, kThreads
// threads each.
__global__ void __launch_bounds__(kThreads, 1)
    ozaki_gemm_kernel(VdvTiles tl, int32_t n_tiles, size_t s_off, VdvColumns cols, int *err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  VdvEpilogue epi{tl, s_off, cols};
  ozaki_tiles(smem, n_tiles, tl.k_tiles, tl, err, epi);
}

// Operators of family blockIdx.y from its plane sums, timeslice t0 +
// blockIdx.z: M = sum_h e^{-2 pi i k h / n_planes} G_h for every k of the
// family.  A thread takes one entry (i, j) and keeps, per distinct |k|, the
// four real sums G.re cos, G.im sin, G.im cos, G.re sin: they give both signs of
// k (for a Hermitian family the entry (j, i) is the conjugate of the sum with
// -k).  Memory-bound: every plane sum is read once, unit stride in i.
constexpr int kMaxK = 4;  // distinct |k| per pass over the planes
__global__ void __launch_bounds__(256)
    vdv_fourier_kernel(double2 *vdv, uint8_t const *scratch, size_t slot_bytes, size_t s_off,
                       VdvFamily const *fams, double2 const *roots, int32_t n_planes,
                       int32_t n_cols, int32_t t0, Geometry g) {
  int const nev = g.nev;
  int64_t const blk = static_cast<int64_t>(nev) * nev;
  int64_t const x = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (x >= blk) return;
  int const i = static_cast<int>(x % nev), j = static_cast<int>(x / nev);
  VdvFamily const &f = fams[blockIdx.y];
  if (f.herm && i > j) return;
  double2 const *G = reinterpret_cast<double2 const *>(scratch + blockIdx.z * slot_bytes + s_off) +
                     static_cast<int64_t>(blockIdx.y) * blk + x;
  int64_t const step = static_cast<int64_t>(n_cols) * nev;
  int const t = t0 + blockIdx.z;
  for (int o0 = 0; o0 < f.n_ops;) {
    // the next operators with at most kMaxK distinct |k|
    int32_t ks[kMaxK];
    int nk = 0, o1 = o0;
#pragma unroll
    for (int q = 0; q < kMaxK; ++q) ks[q] = 0;
    for (; o1 < f.n_ops; ++o1) {
      int32_t const k = abs(f.k[o1]);
      bool known = false;
#pragma unroll
      for (int q = 0; q < kMaxK; ++q) known = known || (q < nk && ks[q] == k);
      if (known) continue;
      if (nk == kMaxK) break;
#pragma unroll
      for (int q = 0; q < kMaxK; ++q)
        if (q == nk) ks[q] = k;
      ++nk;
    }
    double s[kMaxK][4];
    int64_t ph[kMaxK];  // |k| h mod n_planes
#pragma unroll
    for (int q = 0; q < kMaxK; ++q) {
      ph[q] = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) s[q][u] = 0;
      ks[q] %= n_planes;
    }
    for (int h = 0; h < n_planes; ++h) {
      double2 const v = G[h * step];
#pragma unroll
      for (int q = 0; q < kMaxK; ++q) {
        if (q >= nk) break;
        if (ks[q] == 0) {
          s[q][0] += v.x;
          s[q][2] += v.y;
          continue;
        }
        double2 const r = roots[ph[q]];  // (cos, -sin)
        s[q][0] = fma(v.x, r.x, s[q][0]);
        s[q][1] = fma(v.y, -r.y, s[q][1]);
        s[q][2] = fma(v.y, r.x, s[q][2]);
        s[q][3] = fma(v.x, -r.y, s[q][3]);
        ph[q] += ks[q];
        if (ph[q] >= n_planes) ph[q] -= n_planes;
      }
    }
    for (int o = o0; o < o1; ++o) {
      int32_t const k = abs(f.k[o]) % n_planes;
      double u0 = 0, u1 = 0, u2 = 0, u3 = 0;
#pragma unroll
      for (int q = 0; q < kMaxK; ++q)
        if (q < nk && ks[q] == k) {
          u0 = s[q][0];
          u1 = s[q][1];
          u2 = s[q][2];
          u3 = s[q][3];
        }
      if (f.k[o] < 0) {  // e^{+i phi}
        u1 = -u1;
        u3 = -u3;
      }
      double2 *out = vdv + (static_cast<int64_t>(2 * f.op[o]) * g.Lt + t) * blk;
      int64_t const mt = j + static_cast<int64_t>(nev) * i;
      double2 const plus = make_double2(u0 + u1, u2 - u3);  // the sum with k
      if (f.dag[o]) {
        out[mt] = make_double2(plus.x, -plus.y);
      } else {
        out[x] = plus;
        if (f.herm && i != j) out[mt] = make_double2(u0 - u1, -(u2 + u3));
      }
    }
    o0 = o1;
  }
}

struct TcLayout {
  int32_t ktp;
  int64_t k_tiles, n_cols;
  size_t a_bytes, s_off, e_off, n_off, slot_bytes;
};
TcLayout tc_layout(Geometry const &g, VdvTcPlan const &pl) {
  TcLayout L{};
  L.ktp = plane_k_tiles(pl.per);
  L.k_tiles = static_cast<int64_t>(L.ktp) * pl.n_planes;
  int64_t const m_tiles = (2LL * g.nev + kTM - 1) / kTM;
  L.n_cols = pl.cols.n_cols();
  int64_t const n_tiles = (pl.cols.n_all() + kTN - 1) / kTN;
  L.a_bytes = static_cast<size_t>(m_tiles * L.k_tiles) * kStageA;
  L.s_off = L.a_bytes + static_cast<size_t>(n_tiles * L.k_tiles) * kStageB;
  L.e_off = L.s_off + static_cast<size_t>(pl.n_planes * L.n_cols * g.nev) * sizeof(double2);
  // exponents: the eigenvectors', then room for one set per family; norms
  L.n_off = (L.e_off + static_cast<size_t>(1 + pl.n_fam) * g.nev * sizeof(int32_t) + 15) / 16 * 16;
  L.slot_bytes =
      (L.n_off + static_cast<size_t>(g.nev) * sizeof(NormMax) + 1023) / 1024 * 1024;
  return L;
}

}  // namespace

std::vector<int2> vdaggerv_tc_tiles(std::vector<VdvFamily> const &fam, int32_t n_mom,
                                    int32_t nev, int32_t n_planes, int32_t sm_count,
                                    VdvColumns &cols) {
  int32_t const rows = kTM / 2;
  VdvColumns base{nev, static_cast<int32_t>(fam.size()), n_mom, 0, nev};
  while (base.n_lead < n_mom && fam[base.n_lead].herm) ++base.n_lead;
  auto tiles = [&](VdvColumns const &v) {
    std::vector<int2> out;
    for (int64_t nt = 0; nt * kTN < v.n_all(); ++nt)
      for (int32_t mt = 0; mt * rows < nev; ++mt) {
        // wanted: a column (f, j) of the tile with a full family or j >= the tile's
        // first row, and for the rows i >= full none that an edge column stands in for
        bool want = false, last = mt * rows >= v.full;
        for (int64_t c = nt * kTN; c < std::min(v.n_all(), (nt + 1) * kTN) && !want; ++c) {
          int32_t f, j;
          if (v.decode(c, f, j))
            want = !last;
          else
            want = fam[f].herm ? j >= mt * rows : !(last && j < v.full && v.phase(f));
        }
        if (want) out.push_back(make_int2(mt, static_cast<int32_t>(nt)));
      }
    return out;
  };
  cols = base;
  std::vector<int2> out = tiles(base);
  VdvColumns edge = base;
  edge.full = nev / rows * rows;
  if (edge.full > 0 && edge.full < nev && edge.n_all() > edge.n_cols()) {
    // A k-tile of a round of tiles takes 1.3 us, that of one more column's slices
    // 0.1 ns.  Rounds of one timeslice per launch, as streamed eigenvectors have them.
    // 32^3x64 Nev 220, three families (56 columns more, 7 rounds -> 6): GEMM 98.9 ->
    // 86.3 ms, slices 31.5 -> 34.3, pass 171.8 -> 162.2.  24^3x48 Nev 120 (112 more, 2 rounds
    // either way): GEMM 10.0 -> 9.2 but slices 1.4 ms longer, so the plain columns stay.
    std::vector<int2> const e = tiles(edge);
    auto rounds = [&](std::vector<int2> const &t) {
      return (static_cast<int64_t>(t.size()) * n_planes + sm_count - 1) / sm_count;
    };
    int64_t const more = (edge.n_all() - edge.n_cols()) * n_planes;
    if (13000 * (rounds(out) - rounds(e)) > more) {
      cols = edge;
      out = e;
    }
  }
  return out;
}

size_t vdaggerv_tc_scratch_bytes(Geometry g, VdvTcPlan const &pl, int32_t batch) {
  return tc_layout(g, pl).slot_bytes * static_cast<size_t>(batch > 0 ? batch : 1);
}

int32_t vdaggerv_tc_batch(Geometry g, VdvTcPlan const &pl, int32_t sm_count, size_t max_bytes,
                          int32_t n_t) {
  int64_t const per_t = static_cast<int64_t>(pl.n_mn) * pl.n_planes;  // tiles of one timeslice
  int64_t const sms = sm_count > 0 ? sm_count : 1;
  int64_t const nt = n_t > 0 ? n_t : 1;
  int64_t fit = static_cast<int64_t>(max_bytes / tc_layout(g, pl).slot_bytes);
  if (fit > nt) fit = nt;
  if (fit < 1) fit = 1;
  // Persistent CTAs take the tiles of a launch in rounds of one tile per SM;
  // the last round of every launch is partly idle.
  auto rounds = [&](int64_t b) {
    int64_t const launches = (nt + b - 1) / b, last = nt - (launches - 1) * b;
    return (launches - 1) * ((per_t * b + sms - 1) / sms) + (per_t * last + sms - 1) / sms;
  };
  int64_t best = rounds(1);
  for (int64_t b = 2; b <= fit; ++b) best = std::min(best, rounds(b));
  for (int64_t b = 1; b <= fit; ++b)
    if (50 * rounds(b) <= 51 * best) return static_cast<int32_t>(b);
  return static_cast<int32_t>(fit);
}

cudaError_t phase_fixed(longlong2 *phase_fx, double2 const *phase, int64_t n,
                        cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  phase_fixed_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(phase_fx,
                                                                              phase, n);
  return cudaGetLastError();
}

cudaError_t unit_roots(double2 *roots, int32_t n_planes, cudaStream_t stream) {
  unit_roots_kernel<<<(n_planes + 255) / 256, 256, 0, stream>>>(roots, n_planes);
  return cudaGetLastError();
}

cudaError_t vdaggerv_tc(double2 *vdv, double2 const *V, VdvTcPlan const &pl, int32_t t0,
                        int32_t nt, Geometry g, void *scratch, size_t scratch_bytes, int *err,
                        cudaStream_t stream, cudaEvent_t const *t_ready,
                        VdvDisplaced const *disp, cudaEvent_t const *gemm_ev,
                        int32_t n_gemm_ev, int32_t v_t0) {
  int32_t const n_disp = disp ? disp->n : 0;
  if (pl.n_fam == 0 || nt == 0) return cudaSuccess;
  if (pl.n_mom + n_disp != pl.n_fam ||
      (n_disp > 0 && (!disp->n_steps || !disp->steps || !disp->U || !disp->W)))
    return cudaErrorInvalidValue;
  TcLayout const L = tc_layout(g, pl);
  if (L.k_tiles > 0x7fffffffLL / kTK || pl.cols.n_all() > 0x7fffffffLL) return cudaErrorInvalidValue;
  int64_t batch = static_cast<int64_t>(scratch_bytes / L.slot_bytes);
  if (batch < 1) return cudaErrorInvalidValue;
  int64_t const per_t = static_cast<int64_t>(pl.n_mn) * pl.n_planes;
  batch = std::min({batch, std::max<int64_t>(1, 0x7fffffffLL / per_t), int64_t{65535}});
  uint8_t *base = static_cast<uint8_t *>(scratch);
  cudaError_t e = cudaFuncSetAttribute(ozaki_gemm_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(kSmemBytes));
  if (e != cudaSuccess) return e;
  // one warp per (K tile, group of 8 eigenvectors)
  unsigned const sb = static_cast<unsigned>((L.k_tiles * ((g.nev + 7) / 8) * 32 + 255) / 256);
  unsigned const eb = static_cast<unsigned>(
      (L.k_tiles * ((g.nev + 7) / 8 - pl.cols.full / 8) * 32 + 255) / 256);
  unsigned const nc = static_cast<unsigned>((g.dim_row + kNormChunk - 1) / kNormChunk);
  size_t const links = static_cast<size_t>(g.dim_row / 3) * 27;  // of one timeslice
  int32_t const sites = pl.per / 3;
  int64_t const blk = static_cast<int64_t>(g.nev) * g.nev;
  int32_t gemm_k = 0;
  for (int32_t tb = t0; tb < t0 + nt; tb += static_cast<int32_t>(batch)) {
    int32_t const nb = static_cast<int32_t>(std::min<int64_t>(batch, t0 + nt - tb));
    if (t_ready)
      for (int32_t t = tb; t < tb + nb; ++t)
        if (t_ready[t]) {
          e = cudaStreamWaitEvent(stream, t_ready[t], 0);
          if (e != cudaSuccess) return e;
        }
    unsigned const unb = static_cast<unsigned>(nb);
    double2 const *Vb = V + static_cast<int64_t>(tb - v_t0) * g.nev * g.dim_row;
    if (gemm_k == 0) {  // norms start at zero; expo_kernel leaves them so
      e = cudaMemset2DAsync(base + L.n_off, L.slot_bytes, 0,
                            static_cast<size_t>(g.nev) * sizeof(NormMax), unb, stream);
      if (e != cudaSuccess) return e;
    }
    norm_kernel<<<dim3(nc, static_cast<unsigned>(g.nev), unb), 32, 0, stream>>>(base + L.n_off,
                                                                            L.slot_bytes, Vb, g);
    expo_kernel<<<dim3(static_cast<unsigned>(g.nev), unb), 32, 0, stream>>>(
        base + L.n_off, base + L.e_off, L.slot_bytes, Vb, g);
    if (pl.n_mom > 0)
      slice_kernel<true, true, false><<<dim3(sb, unb), 256, 0, stream>>>(
          base, base + L.a_bytes, L.slot_bytes, Vb, pl.phase_fx, pl.n_mom, base + L.e_off,
          pl.n_planes, pl.per, pl.cols, 0, g);
    else
      slice_kernel<true, false, false><<<dim3(sb, unb), 256, 0, stream>>>(
          base, base + L.a_bytes, L.slot_bytes, Vb, nullptr, 0, base + L.e_off, pl.n_planes,
          pl.per, pl.cols, 0, g);
    if (pl.cols.n_all() > pl.cols.n_cols())
      slice_kernel<false, true, true><<<dim3(eb, unb), 256, 0, stream>>>(
          nullptr, base + L.a_bytes, L.slot_bytes, Vb,
          pl.phase_fx + static_cast<int64_t>(pl.cols.n_lead) * sites, pl.n_mom - pl.cols.n_lead,
          base + L.e_off, pl.n_planes, pl.per, pl.cols, pl.cols.n_lead, g);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // Displaced operators: B = D(V_t) with phase 1 and its own column exponents.
    for (int32_t b = 0; b < nb && n_disp > 0; ++b) {
      int32_t const t = tb + b;
      double2 const *Vt = Vb + static_cast<int64_t>(b) * g.nev * g.dim_row;
      uint8_t *slot = base + b * L.slot_bytes;
      for (int32_t d = 0; d < n_disp; ++d) {
        int32_t const f = pl.n_mom + d;
        double2 const *Wt = nullptr;
        e = displaced_vectors(&Wt, disp->W, Vt, disp->U + links * t,
                              disp->P ? disp->P + links * t : nullptr,
                              disp->steps + 2 * static_cast<int64_t>(d) * kMaxDispSteps,
                              disp->n_steps[d], g, stream,
                              reinterpret_cast<NormMax *>(slot + L.n_off));
        if (e != cudaSuccess) return e;
        uint8_t *expo_w = slot + L.e_off + static_cast<size_t>(1 + f) * g.nev * sizeof(int32_t);
        expo_kernel<<<dim3(static_cast<unsigned>(g.nev), 1), 32, 0, stream>>>(slot + L.n_off, expo_w,
                                                                          0, Wt, g);
        slice_kernel<false, true, false><<<dim3(sb, 1), 256, 0, stream>>>(
            nullptr, slot + L.a_bytes, 0, Wt, pl.phase_fx + static_cast<int64_t>(f) * sites, 1,
            expo_w, pl.n_planes, pl.per, pl.cols, f, g);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
      }
    }
    bool const timed = gemm_ev && 2 * gemm_k + 1 < n_gemm_ev;
    if (timed) {
      e = cudaEventRecord(gemm_ev[2 * gemm_k], stream);
      if (e != cudaSuccess) return e;
    }
    VdvTiles const tl{base, L.slot_bytes, L.a_bytes, L.e_off, pl.mn, pl.n_mn, pl.n_planes, L.ktp};
    int64_t const n_tiles = per_t * nb;
    ozaki_gemm_kernel<<<static_cast<unsigned>(persistent_grid(n_tiles)), kThreads, kSmemBytes,
                        stream>>>(tl, static_cast<int32_t>(n_tiles), L.s_off,
                                  pl.cols, err);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (timed) {
      e = cudaEventRecord(gemm_ev[2 * gemm_k + 1], stream);
      if (e != cudaSuccess) return e;
    }
    ++gemm_k;
    vdv_fourier_kernel<<<dim3(static_cast<unsigned>((blk + 255) / 256),
                              static_cast<unsigned>(pl.n_fam), static_cast<unsigned>(nb)),
                         256, 0, stream>>>(vdv, base, L.slot_bytes, L.s_off, pl.fam, pl.roots,
                                           pl.n_planes, static_cast<int32_t>(L.n_cols), tb, g);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

int32_t vdaggerv_tc_gemm_launches(int32_t nt, int32_t batch) {
  return batch > 0 ? (nt + batch - 1) / batch : 0;
}

}  // namespace dev
}  // namespace slaph
