// FP64 kernels of the contraction engine (sm_103a).
//
// Each kernel restates one step of the reference path on the device; the
// reference file:line is given per kernel.  Complex values are double2,
// matrices column-major.
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.cuh"
#include "norm_max.cuh"

namespace slaph {
namespace dev {

namespace {

__constant__ int32_t c_gamma_row[16][4];
__constant__ double2 c_gamma_val[16][4];

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 conjd(double2 a) { return make_double2(a.x, -a.y); }
// acc += a * b
__device__ __forceinline__ void cfma(double2 &acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}
// acc += conj(a) * b
__device__ __forceinline__ void cfmac(double2 &acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, fma(a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(-a.y, b.x, acc.y));
}

// |a| >= |b| as hypot would decide it: the squares settle it unless they are
// within rounding of one another or near the ends of the range (hypot is some
// 50 FP64 operations, five times the rest of a compensated addition).
__device__ __forceinline__ bool not_smaller(double2 a, double2 b) {
  double const p = fma(a.x, a.x, a.y * a.y), q = fma(b.x, b.x, b.y * b.y);
  double const hi = fmax(p, q);
  if (hi > 1e-270 && hi < 1e270 && fabs(p - q) > 1e-14 * hi) return p > q;
  return hypot(a.x, a.y) >= hypot(b.x, b.y);
}

// Neumaier accumulator on complex values, include/KahanAccumulator.hpp:14-48;
// with kahan == 0 it is NativeAccumulator (:50-72).
struct Acc {
  double2 s, c;
  int kahan;
  __device__ explicit Acc(int k) : s(make_double2(0, 0)), c(make_double2(0, 0)), kahan(k) {}
  __device__ void add(double2 x) {
    if (!kahan) {
      s.x += x.x;
      s.y += x.y;
      return;
    }
    double2 const t = make_double2(s.x + x.x, s.y + x.y);
    if (not_smaller(s, x)) {
      c.x += (s.x - t.x) + x.x;
      c.y += (s.y - t.y) + x.y;
    } else {
      c.x += (x.x - t.x) + s.x;
      c.y += (x.y - t.y) + s.y;
    }
    s = t;
  }
  __device__ double2 value() const { return kahan ? make_double2(s.x + c.x, s.y + c.y) : s; }
};

__device__ __forceinline__ int64_t gidx() {
  return blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
}

// ---------------------------------------------------------------- momenta
// create_momenta, src/OperatorFactory.cpp:64-95: exp(-i (px x + py y + pz z)
// 2pi/L) with site index x*Ly*Lz + y*Lz + z.
__global__ void momenta_kernel(double2 *phase, int32_t const *mom, int32_t n_ops, Geometry g) {
  int64_t const vol = static_cast<int64_t>(g.Lx) * g.Ly * g.Lz;
  int64_t const k = gidx();
  if (k >= vol * n_ops) return;
  int const op = static_cast<int>(k / vol);
  int64_t const site = k % vol;
  int const x = static_cast<int>(site / (static_cast<int64_t>(g.Ly) * g.Lz));
  int const y = static_cast<int>((site / g.Lz) % g.Ly);
  int const z = static_cast<int>(site % g.Lz);
  double const ipx = mom[3 * op] * 2. * M_PI / static_cast<double>(g.Lx);
  double const ipy = mom[3 * op + 1] * 2. * M_PI / static_cast<double>(g.Ly);
  double const ipz = mom[3 * op + 2] * 2. * M_PI / static_cast<double>(g.Lz);
  double const arg = (ipx * x + ipy * y) + ipz * z;
  double s, c;
  sincos(arg, &s, &c);
  phase[k] = make_double2(c, -s);
}

// ---------------------------------------------------------------- VdaggerV
// (the build itself: vdv_fp64.cu, vdv_tc.cu)
__global__ void vdv_identity_kernel(double2 *vdv, int32_t op, Geometry g) {
  int64_t const blk = static_cast<int64_t>(g.nev) * g.nev;
  int64_t const k = gidx();
  if (k >= blk * g.Lt) return;
  int64_t const e = k % blk;
  int64_t const t = k / blk;
  double2 const v = make_double2((e % g.nev) == (e / g.nev) ? 1.0 : 0.0, 0.0);
  vdv[(static_cast<int64_t>(2 * op) * g.Lt + t) * blk + e] = v;
  vdv[(static_cast<int64_t>(2 * op + 1) * g.Lt + t) * blk + e] = v;
}

// return_vdaggerv(...).adjoint(), src/DilutedFactorFactory.cpp:53-54.
__global__ void vdv_dagger_kernel(double2 *vdv, int32_t n_ops, Geometry g) {
  int64_t const blk = static_cast<int64_t>(g.nev) * g.nev;
  int64_t const k = gidx();
  if (k >= blk * g.Lt * n_ops) return;
  int64_t const e = k % blk;
  int64_t const rest = k / blk;
  int64_t const t = rest % g.Lt, op = rest / g.Lt;
  int64_t const i = e % g.nev, j = e / g.nev;
  double2 const src = vdv[(2 * op * g.Lt + t) * blk + j + g.nev * i];
  vdv[((2 * op + 1) * g.Lt + t) * blk + e] = conjd(src);
}

// ---------------------------------------------------------------- factors
__device__ __forceinline__ double2 const *vdv_block(double2 const *vdv, int code, int t,
                                                    Geometry const &g) {
  return vdv + (static_cast<int64_t>(code) * g.Lt + t) * g.nev * static_cast<int64_t>(g.nev);
}
__device__ __forceinline__ double2 rnd(double2 const *noise, int r, int64_t blk,
                                       Geometry const &g) {
  return noise[static_cast<int64_t>(r) * g.Lt * 4 * g.nev + blk];
}
__device__ __forceinline__ int64_t peram_rows(Geometry const &g) {
  return 4LL * g.nev * g.Lt;
}
__device__ __forceinline__ double2 const *peram_of(double2 const *peram, int r,
                                                   Geometry const &g) {
  return peram + static_cast<int64_t>(r) * peram_rows(g) * g.nb * 4 * g.dilE;
}

// Q0 intermediate, src/DilutedFactorFactory.cpp:66-78:
// M[v, e + dilE d] = sum_{w = e mod dilE} rho_r2[d + 4(w + nev t)] vdv[v, w].
__global__ void q0m_kernel(double2 *out, Q0MInst const *inst, double2 const *vdv,
                           double2 const *noise, Geometry g) {
  Q0MInst const in = inst[blockIdx.y];
  int const nev = g.nev, eds = 4 * g.dilE;
  int const k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nev * eds) return;
  int const v = k % nev, c = k / nev;
  int const e = c % g.dilE, d = c / g.dilE;
  double2 const *m = vdv_block(vdv, in.vdv, in.t, g);
  double2 acc = make_double2(0, 0);
  for (int w = e; w < nev; w += g.dilE)
    cfma(acc, rnd(noise, in.r2, d + 4 * (w + static_cast<int64_t>(nev) * in.t), g),
         m[v + static_cast<int64_t>(nev) * w]);
  out[static_cast<int64_t>(blockIdx.y) * nev * eds + k] = acc;
}

// Q1 intermediate, src/DilutedFactorFactory.cpp:134-144:
// R[e + dilE d, j] = sum_{v = e mod dilE} conj(rho_r1[d + 4 v + 4 nev t]) vdv[v, j].
__global__ void q1r_kernel(double2 *out, Q1RInst const *inst, double2 const *vdv,
                           double2 const *noise, Geometry g) {
  Q1RInst const in = inst[blockIdx.y];
  int const nev = g.nev, eds = 4 * g.dilE;
  int const k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nev * eds) return;
  int const a = k % eds, j = k / eds;
  int const e = a % g.dilE, d = a / g.dilE;
  double2 const *m = vdv_block(vdv, in.vdv, in.t, g);
  double2 acc = make_double2(0, 0);
  for (int v = e; v < nev; v += g.dilE)
    cfmac(acc, rnd(noise, in.r1, d + 4 * (v + static_cast<int64_t>(nev) * in.t), g),
          m[v + static_cast<int64_t>(nev) * j]);
  out[static_cast<int64_t>(blockIdx.y) * nev * eds + k] = acc;
}

// Q2 intermediate, src/DilutedFactorFactory.cpp:203-218 (without the gamma_5
// signs, applied in q2_kernel):
// M[col dilE + e, row nev + v] = sum_w conj(P_r1[(4t + row) nev + w,
//                                               (4 b1 + col) dilE + e]) vdv[w, v].
// Per CTA a 32 x 64 tile of the rows (dirac row, a) of all four Dirac blocks, so
// that only the last of 4 eds / 32 tiles has padding; 16 w per step.
constexpr int MT = 32, NT = 64, KT = 16;
__global__ void __launch_bounds__(256) q2m_kernel(double2 *out, Q2MInst const *inst,
                                                  double2 const *vdv, double2 const *peram,
                                                  Geometry g) {
  __shared__ double2 As[KT][MT + 1];
  __shared__ double2 Bs[KT][NT];
  Q2MInst const in = inst[blockIdx.y];
  int const nev = g.nev, eds = 4 * g.dilE;
  int const ntile = (nev + NT - 1) / NT;
  int const v0 = (blockIdx.x % ntile) * NT;
  int const m0 = (blockIdx.x / ntile) * MT;
  int const tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  int64_t const rows = peram_rows(g);
  double2 const *P = peram_of(peram, in.r1, g) + static_cast<int64_t>(4 * in.t) * nev +
                     rows * (static_cast<int64_t>(in.b1) * eds);
  double2 const *m = vdv_block(vdv, in.vdv, in.t, g);
  // Rows that this thread stages, and whether its outputs are wanted at all
  // (warps without any skip the arithmetic).
  double2 const *row_p[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    int const mm = m0 + tid / KT + 16 * q;
    row_p[q] = mm < 4 * eds ? P + static_cast<int64_t>(mm / eds) * nev + rows * (mm % eds) : nullptr;
  }
  bool const warp_on = m0 + (ty & ~1) < 4 * eds;
  double2 acc[2][4];
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[p][q] = make_double2(0, 0);
  for (int w0 = 0; w0 < nev; w0 += KT) {
    int const wk = w0 + tid % KT;
#pragma unroll
    for (int q = 0; q < 2; ++q)
      As[tid % KT][tid / KT + 16 * q] =
          wk < nev && row_p[q] ? row_p[q][wk] : make_double2(0, 0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int const k = tid + 256 * q;
      int const ww = k % KT, vv = k / KT;
      int const w = w0 + ww, v = v0 + vv;
      Bs[ww][vv] = (w < nev && v < nev) ? m[w + static_cast<int64_t>(nev) * v]
                                        : make_double2(0, 0);
    }
    __syncthreads();
    if (warp_on)
#pragma unroll 4
      for (int kk = 0; kk < KT; ++kk) {
        double2 a[2], b[4];
#pragma unroll
        for (int p = 0; p < 2; ++p) a[p] = As[kk][ty + 16 * p];
#pragma unroll
        for (int q = 0; q < 4; ++q) b[q] = Bs[kk][tx + 16 * q];
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int q = 0; q < 4; ++q) cfmac(acc[p][q], a[p], b[q]);
      }
    __syncthreads();
  }
  double2 *o = out + static_cast<int64_t>(blockIdx.y) * eds * 4 * nev;
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int const mm = m0 + ty + 16 * p, v = v0 + tx + 16 * q;
      if (mm < 4 * eds && v < nev)
        o[mm % eds + static_cast<int64_t>(eds) * (mm / eds * nev + v)] = acc[p][q];
    }
}

// Q0 factor, src/DilutedFactorFactory.cpp:80-98:
// Q0[e1 + dilE g, d dilE + e2] = val[d] sum_{v = e1} M[v, d dilE + e2]
//                                conj(rho_r1[g + 4(v + nev t)]),  g = row[d].
__global__ void q0_kernel(double2 *slots, Q0Inst const *inst, double2 const *q0m,
                          double2 const *noise, Geometry g) {
  Q0Inst const in = inst[blockIdx.y];
  int const nev = g.nev, dilE = g.dilE, eds = 4 * dilE;
  int const k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= eds * eds) return;
  int const a = k % eds, b = k / eds;
  int const d = b / dilE;
  int const gr = c_gamma_row[in.gamma][d];
  double2 acc = make_double2(0, 0);
  if (a / dilE == gr) {
    int const e1 = a % dilE;
    double2 const *M = q0m + static_cast<int64_t>(in.m) * nev * eds;
    double2 const val = c_gamma_val[in.gamma][d];
    for (int v = e1; v < nev; v += dilE) {
      double2 const vm = cmul(val, M[v + static_cast<int64_t>(nev) * b]);
      double2 const cr =
          conjd(rnd(noise, in.r1, gr + 4 * (v + static_cast<int64_t>(nev) * in.t), g));
      cfma(acc, vm, cr);
    }
  }
  slots[static_cast<int64_t>(in.slot) * eds * eds + k] = acc;
}

// Q1 factor, src/DilutedFactorFactory.cpp:146-164:
// Q1[row dilE + e, col dilE + f] = val[row] sum_v R[row dilE + e, v]
//        P_r2[(4t + grow[row]) nev + v, (4b + col) dilE + f].
__global__ void q1_kernel(double2 *slots, Q1Inst const *inst, double2 const *q1r,
                          double2 const *peram, Geometry g) {
  Q1Inst const in = inst[blockIdx.y];
  int const nev = g.nev, dilE = g.dilE, eds = 4 * dilE;
  int const k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= eds * eds) return;
  int const a = k % eds, c = k / eds;
  int const row = a / dilE;
  int64_t const rows = peram_rows(g);
  double2 const *R = q1r + static_cast<int64_t>(in.r) * nev * eds;
  double2 const *P = peram_of(peram, in.r2, g) +
                     static_cast<int64_t>(4 * in.t + c_gamma_row[in.gamma][row]) * nev +
                     rows * (static_cast<int64_t>(in.b) * eds + c);
  double2 acc = make_double2(0, 0);
  for (int v = 0; v < nev; ++v) cfma(acc, R[a + static_cast<int64_t>(eds) * v], P[v]);
  slots[static_cast<int64_t>(in.slot) * eds * eds + k] = cmul(c_gamma_val[in.gamma][row], acc);
}

// The products R P_r2 of all four Dirac blocks d of the perambulator, shared by
// the Q1 factors that differ in gamma only: X[a, d eds + c] = sum_v R[a, v]
// P_r2[(4t + d) nev + v, b eds + c], summed as in q1_kernel.  One CTA per
// instance and Dirac block.
__global__ void x1_kernel(double2 *out, X1Inst const *inst, double2 const *q1r,
                          double2 const *peram, Geometry g) {
  X1Inst const in = inst[blockIdx.y];
  int const nev = g.nev, eds = 4 * g.dilE;
  int const k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= 4 * eds * eds) return;
  int const a = k % eds, c = k / eds % eds, d = k / (eds * eds);
  int64_t const rows = peram_rows(g);
  double2 const *R = q1r + static_cast<int64_t>(in.r) * nev * eds + a;
  double2 const *P = peram_of(peram, in.r2, g) + static_cast<int64_t>(4 * in.t + d) * nev +
                     rows * (static_cast<int64_t>(in.b) * eds + c);
  double2 acc = make_double2(0, 0);
  for (int v = 0; v < nev; ++v) cfma(acc, R[static_cast<int64_t>(eds) * v], P[v]);
  out[static_cast<int64_t>(blockIdx.y) * 4 * eds * eds + k] = acc;
}

// Q1 factors from those products: val[row] X[a, Grow[row] eds + c].
__global__ void q1_pick_kernel(double2 *slots, Q1Pick const *inst, double2 const *x, int32_t dilE) {
  Q1Pick const in = inst[blockIdx.y];
  int const eds = 4 * dilE;
  int const k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= eds * eds) return;
  int const row = k % eds / dilE;
  double2 const v = x[(4LL * in.x + c_gamma_row[in.gamma][row]) * eds * eds + k];
  slots[static_cast<int64_t>(in.slot) * eds * eds + k] = cmul(c_gamma_val[in.gamma][row], v);
}

// Q2 factor, src/DilutedFactorFactory.cpp:214-243:
// Q2[r dilE + e, col dilE + f] = sum_bd val[bd] s(bd, r)
//     sum_v M[r dilE + e, bd nev + v] P_r2[(4t + grow[bd]) nev + v, (4 b2 + col) dilE + f]
// with the gamma_5 sign s = -1 when bd + r == 3 or |bd - r| > 1 (:215-216).
__global__ void q2_kernel(double2 *slots, Q2Inst const *inst, double2 const *q2m,
                          double2 const *peram, Geometry g) {
  Q2Inst const in = inst[blockIdx.y];
  int const nev = g.nev, dilE = g.dilE, eds = 4 * dilE;
  int const k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= eds * eds) return;
  int const a = k % eds, c = k / eds;
  int const r = a / dilE;
  int64_t const rows = peram_rows(g);
  double2 const *M = q2m + static_cast<int64_t>(in.m) * eds * 4 * nev;
  double2 const *Pr = peram_of(peram, in.r2, g) + rows * (static_cast<int64_t>(in.b2) * eds + c);
  double2 total = make_double2(0, 0);
  for (int bd = 0; bd < 4; ++bd) {
    double2 const *P = Pr + static_cast<int64_t>(4 * in.t + c_gamma_row[in.gamma][bd]) * nev;
    double2 const *Mb = M + a + static_cast<int64_t>(eds) * bd * nev;
    double2 acc = make_double2(0, 0);
    for (int v = 0; v < nev; ++v) cfma(acc, Mb[static_cast<int64_t>(eds) * v], P[v]);
    bool const flip = (bd + r == 3) || (bd - r > 1) || (r - bd > 1);
    double2 const val = c_gamma_val[in.gamma][bd];
    double2 const s = flip ? make_double2(-val.x, -val.y) : val;
    double2 const pr = cmul(s, acc);
    total.x += pr.x;
    total.y += pr.y;
  }
  slots[static_cast<int64_t>(in.slot) * eds * eds + k] = total;
}

// ---------------------------------------------------------------- products
// operator*(vector<DF>, vector<DF>) data part, src/DilutedFactor.cpp:40-41:
// C = A * B for eds x eds matrices; one CTA per product, operands in smem.
__global__ void __launch_bounds__(256) product_kernel(double2 *slots, ProdInst const *p,
                                                      int32_t eds) {
  extern __shared__ double2 sm[];
  ProdInst const in = p[blockIdx.x];
  int64_t const ms = static_cast<int64_t>(eds) * eds;
  double2 *As = sm, *Bs = sm + ms;
  double2 const *A = slots + in.a * ms;
  double2 const *B = slots + in.b * ms;
  for (int k = threadIdx.x; k < ms; k += blockDim.x) {
    As[k] = A[k];
    Bs[k] = B[k];
  }
  __syncthreads();
  double2 *C = slots + in.c * ms;
  for (int k = threadIdx.x; k < ms; k += blockDim.x) {
    int const i = k % eds, j = k / eds;
    double2 acc = make_double2(0, 0);
    for (int q = 0; q < eds; ++q) cfma(acc, As[i + eds * q], Bs[q + eds * j]);
    C[k] = acc;
  }
}

// ---------------------------------------------------------------- traces
// factor_to_trace, src/DilutedTrace.cpp:84-165: tr(L R) per entry (or tr(F)).
// One CTA per list, one lane per row; a warp takes 32 / eds entries at once when
// the matrices have 16 rows or fewer (16 rows left half of its lanes idle:
// 4^3x8 pipi set at eds 16, 5.2 -> 2.6 ms).
__global__ void __launch_bounds__(256) trace_kernel(double2 *values, TraceList const *lists,
                                                    int32_t const *which,
                                                    int32_t const *shape_i,
                                                    int32_t const *shape_j,
                                                    int64_t const *shape_off,
                                                    double2 const *slots, int32_t eds) {
  TraceList const L = lists[which[blockIdx.x]];
  int64_t const off = shape_off[L.shape];
  int const n = static_cast<int>(shape_off[L.shape + 1] - off);
  int const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  int const per = eds <= 16 ? 32 / eds : 1;  // entries per warp
  int const sub = per > 1 ? lane / eds : 0, i0 = per > 1 ? lane % eds : lane;
  int64_t const ms = static_cast<int64_t>(eds) * eds;
  for (int e0 = warp * per; e0 < n; e0 += blockDim.x / 32 * per) {
    int const e = e0 + sub;
    bool const on = sub < per && e < n;
    int const ia = on ? shape_i[off + e] : 0, jb = on ? shape_j[off + e] : -1;
    double2 const *A = slots + (static_cast<int64_t>(L.a_base) + ia) * ms;
    double2 acc = make_double2(0, 0);
    if (on && jb >= 0) {
      double2 const *B = slots + (static_cast<int64_t>(L.b_base) + jb) * ms;
      for (int i = i0; i < eds; i += 32) {
        double2 row = make_double2(0, 0);
        for (int j = 0; j < eds; ++j) cfma(row, A[i + eds * j], B[j + eds * i]);
        acc.x += row.x;
        acc.y += row.y;
      }
    } else if (on) {
      for (int i = i0; i < eds; i += 32) {
        acc.x += A[i + eds * i].x;
        acc.y += A[i + eds * i].y;
      }
    }
    // sum over the lanes of an entry (rows i0 + s beyond its last add nothing)
    int const width = per > 1 ? eds : 32;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      double const x = __shfl_down_sync(0xffffffffu, acc.x, s);
      double const y = __shfl_down_sync(0xffffffffu, acc.y, s);
      if (i0 + s < width) {
        acc.x += x;
        acc.y += y;
      }
    }
    if (on && i0 == 0) values[L.val_off + static_cast<int64_t>(e) * L.stride] = acc;
  }
}

// ---------------------------------------------------------------- terms
// resolve_request1/2/3 (src/Diagram.cpp:9-94) with inner_product
// (src/DilutedTrace.cpp:5-82): one thread per (request, slice pair), the
// reference's loop order and accumulator.  The FP64 units bound it.  The inner
// sum of a product of two traces depends on the outer entry's random-vector mask
// only, which ordered index tuples share (two orders of a pair, six of three), so
// the sums of the first kTermMemo outer entries are kept and taken again.
constexpr int kTermMemo = 32;
__global__ void term_kernel(double2 *term_val, Term const *terms, int64_t n,
                            TraceList const *lists, double2 const *values,
                            uint16_t const *shape_mask, int64_t const *shape_off,
                            int32_t kahan) {
  int64_t const k = gidx();
  if (k >= n) return;
  Term const t = terms[k];
  TraceList const L0 = lists[t.list[0]];
  int64_t const o0 = shape_off[L0.shape];
  int64_t const n0 = shape_off[L0.shape + 1] - o0;
  double2 const *x0 = values + L0.val_off;
  int64_t const s0 = L0.stride;
  uint16_t const *m0 = shape_mask + o0;
  double2 res;
  if (t.n == 1) {
    Acc a(kahan);
    for (int64_t e = 0; e < n0; ++e) a.add(x0[e * s0]);
    double2 const v = a.value();
    res = make_double2(v.x / static_cast<double>(n0), v.y / static_cast<double>(n0));
  } else {
    TraceList const L1 = lists[t.list[1]];
    int64_t const o1 = shape_off[L1.shape];
    int64_t const n1 = shape_off[L1.shape + 1] - o1;
    double2 const *x1 = values + L1.val_off;
    int64_t const s1 = L1.stride;
    uint16_t const *m1 = shape_mask + o1;
    int64_t num = 0;
    Acc result(kahan);
    if (t.n == 2) {
      double2 memo[kTermMemo];
      int32_t memo_n[kTermMemo];
      for (int64_t l = 0; l < n0; ++l) {
        uint16_t const m = m0[l];
        int f = 0;  // the first entry with this mask
        while (f < l && f < kTermMemo && m0[f] != m) ++f;
        bool const again = f < l && f < kTermMemo;
        double2 inner = make_double2(0, 0);
        int32_t cnt = 0;
        if (again) {
          inner = memo[f];
          cnt = memo_n[f];
        } else {
          Acc rs(kahan);
          for (int64_t r = 0; r < n1; ++r) {
            if ((m & m1[r]) != 0u) continue;
            rs.add(x1[r * s1]);
            ++cnt;
          }
          inner = rs.value();
          if (l < kTermMemo) {
            memo[l] = inner;
            memo_n[l] = cnt;
          }
        }
        num += cnt;
        result.add(cmul(x0[l * s0], inner));
      }
    } else {
      TraceList const L2 = lists[t.list[2]];
      int64_t const o2 = shape_off[L2.shape];
      int64_t const n2 = shape_off[L2.shape + 1] - o2;
      double2 const *x2 = values + L2.val_off;
      int64_t const s2 = L2.stride;
      uint16_t const *m2 = shape_mask + o2;
      for (int64_t l = 0; l < n0; ++l)
        for (int64_t m = 0; m < n1; ++m) {
          Acc rs(kahan);
          for (int64_t r = 0; r < n2; ++r) {
            if ((m0[l] & m1[m] & m2[r]) != 0u) continue;
            rs.add(x2[r * s2]);
            ++num;
          }
          result.add(cmul(cmul(x0[l * s0], x1[m * s1]), rs.value()));
        }
    }
    double2 const v = result.value();
    double const dn = static_cast<double>(num);
    res = num ? make_double2(v.x / dn, v.y / dn) : make_double2(0, 0);
  }
  term_val[k] = res;
}

// Diagram::assemble (src/Diagram.cpp:96-114): correlator[dt][i] += c in the
// order the terms were produced.
__global__ void accumulate_kernel(double2 *running, int32_t const *seg_out,
                                  int64_t const *seg_off, int64_t n_seg, int32_t const *idx,
                                  double2 const *term_val) {
  int64_t const s = gidx();
  if (s >= n_seg) return;
  double2 acc = running[seg_out[s]];
  for (int64_t k = seg_off[s]; k < seg_off[s + 1]; ++k) {
    double2 const v = term_val[idx[k]];
    acc.x += v.x;
    acc.y += v.y;
  }
  running[seg_out[s]] = acc;
}

__global__ void divide_kernel(double2 *x, int64_t n, double d) {
  int64_t const k = gidx();
  if (k < n) x[k] = make_double2(x[k].x / d, x[k].y / d);
}

int blocks_for(int64_t n, int threads) {
  return static_cast<int>((n + threads - 1) / threads);
}

}  // namespace

// The gamma table of src/Gamma.cpp:18-246 (tmLQCD basis): for matrix m and
// column c the non-zero row and its value (+-1, +-i).
namespace {
// Gamma table (the data of src/Gamma.cpp:18-246): Gamma_m has, in column c, its
// single nonzero at row kGammaRow[m][c] with value kGammaVal[m][c] (re, im).
int32_t const kGammaRow[16][4] = {{2, 3, 0, 1}, {3, 2, 1, 0}, {3, 2, 1, 0}, {2, 3, 0, 1},
                                  {0, 1, 2, 3}, {0, 1, 2, 3}, {2, 3, 0, 1}, {3, 2, 1, 0},
                                  {3, 2, 1, 0}, {2, 3, 0, 1}, {1, 0, 3, 2}, {1, 0, 3, 2},
                                  {0, 1, 2, 3}, {1, 0, 3, 2}, {1, 0, 3, 2}, {0, 1, 2, 3}};
double const kGammaVal[16][4][2] = {
    {{1, 0}, {1, 0}, {1, 0}, {1, 0}},      {{0, -1}, {0, -1}, {0, 1}, {0, 1}},
    {{1, 0}, {-1, 0}, {-1, 0}, {1, 0}},    {{0, -1}, {0, 1}, {0, 1}, {0, -1}},
    {{1, 0}, {1, 0}, {1, 0}, {1, 0}},      {{1, 0}, {1, 0}, {-1, 0}, {-1, 0}},
    {{1, 0}, {1, 0}, {-1, 0}, {-1, 0}},    {{0, -1}, {0, -1}, {0, -1}, {0, -1}},
    {{1, 0}, {-1, 0}, {1, 0}, {-1, 0}},    {{0, -1}, {0, 1}, {0, -1}, {0, 1}},
    {{0, -1}, {0, -1}, {0, 1}, {0, 1}},    {{1, 0}, {-1, 0}, {-1, 0}, {1, 0}},
    {{0, -1}, {0, 1}, {0, 1}, {0, -1}},    {{0, -1}, {0, -1}, {0, -1}, {0, -1}},
    {{1, 0}, {-1, 0}, {1, 0}, {-1, 0}},    {{0, -1}, {0, 1}, {0, -1}, {0, 1}}};
}  // namespace

int32_t gamma_row_host(int32_t m, int32_t c) { return kGammaRow[m][c]; }
int32_t gamma_phase_host(int32_t m, int32_t c) {
  double const re = kGammaVal[m][c][0], im = kGammaVal[m][c][1];
  return re > 0 ? 0 : im > 0 ? 1 : re < 0 ? 2 : 3;
}

cudaError_t upload_gamma(cudaStream_t stream) {
  double2 v[16][4];
  for (int m = 0; m < 16; ++m)
    for (int c = 0; c < 4; ++c) v[m][c] = make_double2(kGammaVal[m][c][0], kGammaVal[m][c][1]);
  cudaError_t e = cudaMemcpyToSymbolAsync(c_gamma_row, kGammaRow, sizeof kGammaRow, 0,
                                          cudaMemcpyHostToDevice, stream);
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbolAsync(c_gamma_val, v, sizeof v, 0, cudaMemcpyHostToDevice, stream);
}

cudaError_t momenta(double2 *phase, int32_t const *mom, int32_t n_ops, Geometry g,
                    cudaStream_t stream) {
  int64_t const n = static_cast<int64_t>(g.Lx) * g.Ly * g.Lz * n_ops;
  if (n == 0) return cudaSuccess;
  momenta_kernel<<<blocks_for(n, 256), 256, 0, stream>>>(phase, mom, n_ops, g);
  return cudaGetLastError();
}

// displace_eigenvectors (src/OperatorFactory.cpp:33-55) for one step on a
// cubic lattice.  The reference updates its copy in place, each line of the
// step's direction in increasing site index, so a site reads the
// already-displaced value of a preceding neighbour.  Forward, W(c) = U(c) V(c +
// 1) for the sites c of a line, only the last site wraps to one: W(L - 1) =
// U(L - 1) W(0).  Backward, W(c) = U(c - 1)^H W(c - 1) with W(0) = U(L - 1)^H
// V(L - 1), every site is a product of links applied to V(L - 1): W(c) = P(c)
// V(L - 1), P(0) = U(L - 1)^H, P(c) = U(c - 1)^H P(c - 1) (forward_uv /
// backward_uv, src/GaugeField.cpp:543-560).  Out of place, all sites are
// independent; P does not depend on the eigenvector and is formed once per
// timeslice (line_products, all timeslices in one launch: a line is a serial
// chain of L products: 105 us for one timeslice at 24^3, 440 us for 48).

namespace {

struct Line {
  int64_t base, stride;
  int c;
};
__device__ __forceinline__ Line line_of(int64_t s, int dir, int L) {
  int64_t const stride = dir == 0 ? static_cast<int64_t>(L) * L : dir == 1 ? L : 1;
  int const c = static_cast<int>(s / stride % L);
  return {s - c * stride, stride, c};
}

// P(c) of every line of direction blockIdx.y and timeslice blockIdx.z, one
// thread per line: [t][site][dir][a + 3 b].
__global__ void line_product_kernel(double2 *P, double2 const *U, int32_t L) {
  int64_t const lines = static_cast<int64_t>(L) * L;
  int64_t const l = gidx();
  int const dir = blockIdx.y;
  if (l >= lines) return;
  P += blockIdx.z * lines * L * 27;
  U += blockIdx.z * lines * L * 27;
  int64_t const stride = dir == 0 ? lines : dir == 1 ? L : 1;
  int64_t const base = dir == 0 ? l : dir == 1 ? (l / L) * lines + l % L : l * L;
  double2 p[9], u[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) p[k] = make_double2(k % 4 == 0 ? 1.0 : 0.0, 0.0);
  for (int c = 0; c < L; ++c) {
    double2 const *src = U + ((base + (c + L - 1) % L * stride) * 3 + dir) * 9;
#pragma unroll
    for (int k = 0; k < 9; ++k) u[k] = src[k];
    double2 *dst = P + ((base + c * stride) * 3 + dir) * 9;
    double2 r[9];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        double2 acc = make_double2(0, 0);
#pragma unroll
        for (int k = 0; k < 3; ++k) cfmac(acc, u[k + 3 * a], p[k + 3 * b]);
        r[a + 3 * b] = acc;
        dst[a + 3 * b] = acc;
      }
#pragma unroll
    for (int k = 0; k < 9; ++k) p[k] = r[k];
  }
}

// One thread per site, kDispEv eigenvectors with the site's matrix in
// registers.  Bound by FP64 issue (36 multiply-adds per site and eigenvector);
// the largest norms of the columns (norms, when given: see NormMax) are integer
// and FP32 work beside it.
constexpr int kDispEv = 8;
__global__ void __launch_bounds__(128)
    displace_kernel(double2 *W, double2 const *V, double2 const *M, int32_t dir, int32_t forward,
                    NormMax *norms, Geometry g) {
  int const L = g.Lx;
  bool const on = gidx() < g.dim_row / 3;  // (no early return: warp reductions below)
  int64_t const s = on ? gidx() : 0;
  Line const ln = line_of(s, dir, L);
  double2 m[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) m[k] = M[(s * 3 + dir) * 9 + k];
  bool const wrap = forward && ln.c + 1 == L && L > 1;
  int64_t const from = forward ? ln.base + (wrap ? 1 : (ln.c + 1) % L) * ln.stride
                               : ln.base + (L - 1) * ln.stride;
  if (wrap) {  // U(L - 1) U(0), applied to V(1)
    double2 const *u0 = M + (ln.base * 3 + dir) * 9;
    double2 r[9];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        double2 acc = make_double2(0, 0);
#pragma unroll
        for (int k = 0; k < 3; ++k) cfma(acc, m[a + 3 * k], u0[k + 3 * b]);
        r[a + 3 * b] = acc;
      }
#pragma unroll
    for (int k = 0; k < 9; ++k) m[k] = r[k];
  }
  int const e0 = blockIdx.y * kDispEv, e1 = min(g.nev, e0 + kDispEv);
  for (int ev = e0; ev < e1; ++ev) {
    double2 const *src = V + ev * g.dim_row + 3 * from;
    double2 v[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) v[b] = src[b];
    double2 *dst = W + ev * g.dim_row + 3 * s;
    NormMax nm{0, 0};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      double2 acc = make_double2(0, 0);
#pragma unroll
      for (int b = 0; b < 3; ++b) cfma(acc, m[a + 3 * b], v[b]);
      if (on) dst[a] = acc;
      norm_max(nm, acc);
    }
    if (norms) norm_max_add(norms + ev, nm);
  }
}

}  // namespace

cudaError_t line_products(double2 *P, double2 const *U, Geometry g, cudaStream_t stream) {
  if (g.Lx != g.Ly || g.Lx != g.Lz) return cudaErrorInvalidValue;
  int64_t const lines = static_cast<int64_t>(g.Lx) * g.Lx;
  for (int32_t t = 0; t < g.Lt; t += 65535) {
    int64_t const at = t * lines * g.Lx * 27;
    line_product_kernel<<<dim3(blocks_for(lines, 32), 3, g.Lt - t < 65535 ? g.Lt - t : 65535), 32,
                          0, stream>>>(P + at, U + at, g.Lx);
  }
  return cudaGetLastError();
}

namespace {
cudaError_t displace(double2 *W, double2 const *V, double2 const *U, double2 const *P,
                     int32_t dir, int32_t forward, NormMax *norms, Geometry g,
                     cudaStream_t stream) {
  if (dir < 0 || dir > 2 || g.Lx != g.Ly || g.Lx != g.Lz) return cudaErrorInvalidValue;
  displace_kernel<<<dim3(blocks_for(g.dim_row / 3, 128), blocks_for(g.nev, kDispEv)), 128, 0,
                    stream>>>(W, V, forward ? U : P, dir, forward, norms, g);
  return cudaGetLastError();
}
}  // namespace

cudaError_t displaced_vectors(double2 const **out, double2 *W, double2 const *V, double2 const *U,
                              double2 const *P, int32_t const *steps, int32_t n, Geometry g,
                              cudaStream_t stream, NormMax *norms) {
  int64_t const n_v = static_cast<int64_t>(g.nev) * g.dim_row;
  double2 const *src = V;
  for (int32_t k = 0; k < n; ++k) {
    double2 *dst = W + (k % 2) * n_v;
    cudaError_t const e = displace(dst, src, U, P, steps[2 * k], steps[2 * k + 1],
                                   k + 1 == n ? norms : nullptr, g, stream);
    if (e != cudaSuccess) return e;
    src = dst;
  }
  *out = src;
  return cudaSuccess;
}

cudaError_t vdaggerv_identity(double2 *vdv, int32_t op, Geometry g, cudaStream_t stream) {
  int64_t const n = static_cast<int64_t>(g.nev) * g.nev * g.Lt;
  vdv_identity_kernel<<<blocks_for(n, 256), 256, 0, stream>>>(vdv, op, g);
  return cudaGetLastError();
}

cudaError_t vdaggerv_daggers(double2 *vdv, int32_t n_ops, Geometry g, cudaStream_t stream) {
  int64_t const n = static_cast<int64_t>(g.nev) * g.nev * g.Lt * n_ops;
  if (n == 0) return cudaSuccess;
  vdv_dagger_kernel<<<blocks_for(n, 256), 256, 0, stream>>>(vdv, n_ops, g);
  return cudaGetLastError();
}

// Grids over instances are split in chunks of 65535 (gridDim.y limit).
template <typename Inst, typename F>
cudaError_t chunked(Inst const *inst, int64_t n, F &&launch) {
  for (int64_t s = 0; s < n; s += 65535) {
    int const c = static_cast<int>(n - s < 65535 ? n - s : 65535);
    launch(inst + s, c, s);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t q0m(double2 *out, Q0MInst const *inst, int64_t n, double2 const *vdv,
                double2 const *noise, Geometry g, cudaStream_t stream) {
  int64_t const per = static_cast<int64_t>(g.nev) * 4 * g.dilE;
  return chunked(inst, n, [&](Q0MInst const *p, int c, int64_t s) {
    q0m_kernel<<<dim3(blocks_for(per, 256), c), 256, 0, stream>>>(out + s * per, p, vdv, noise, g);
  });
}

cudaError_t q1r(double2 *out, Q1RInst const *inst, int64_t n, double2 const *vdv,
                double2 const *noise, Geometry g, cudaStream_t stream) {
  int64_t const per = static_cast<int64_t>(g.nev) * 4 * g.dilE;
  return chunked(inst, n, [&](Q1RInst const *p, int c, int64_t s) {
    q1r_kernel<<<dim3(blocks_for(per, 256), c), 256, 0, stream>>>(out + s * per, p, vdv, noise, g);
  });
}

cudaError_t q2m(double2 *out, Q2MInst const *inst, int64_t n, double2 const *vdv,
                double2 const *peram, Geometry g, cudaStream_t stream) {
  int const eds = 4 * g.dilE;
  int64_t const per = static_cast<int64_t>(eds) * 4 * g.nev;
  int const ntile = (g.nev + NT - 1) / NT, mtile = (4 * eds + MT - 1) / MT;
  return chunked(inst, n, [&](Q2MInst const *p, int c, int64_t s) {
    q2m_kernel<<<dim3(ntile * mtile, c), 256, 0, stream>>>(out + s * per, p, vdv, peram, g);
  });
}

cudaError_t q0(double2 *slots, Q0Inst const *inst, int64_t n, double2 const *q0m_,
               double2 const *noise, Geometry g, cudaStream_t stream) {
  int64_t const per = 16LL * g.dilE * g.dilE;
  return chunked(inst, n, [&](Q0Inst const *p, int c, int64_t) {
    q0_kernel<<<dim3(blocks_for(per, 256), c), 256, 0, stream>>>(slots, p, q0m_, noise, g);
  });
}

cudaError_t q1(double2 *slots, Q1Inst const *inst, int64_t n, double2 const *q1r_,
               double2 const *peram, Geometry g, cudaStream_t stream) {
  int64_t const per = 16LL * g.dilE * g.dilE;
  return chunked(inst, n, [&](Q1Inst const *p, int c, int64_t) {
    q1_kernel<<<dim3(blocks_for(per, 256), c), 256, 0, stream>>>(slots, p, q1r_, peram, g);
  });
}

cudaError_t q1_shared(double2 *slots, double2 *x, X1Inst const *xi, int64_t n_x,
                      Q1Pick const *picks, int64_t n, double2 const *q1r_, double2 const *peram,
                      Geometry g, cudaStream_t stream) {
  int64_t const per = 16LL * g.dilE * g.dilE;
  cudaError_t const e = chunked(xi, n_x, [&](X1Inst const *p, int c, int64_t s) {
    x1_kernel<<<dim3(blocks_for(4 * per, 256), c), 256, 0, stream>>>(x + s * 4 * per, p, q1r_,
                                                                     peram, g);
  });
  if (e != cudaSuccess) return e;
  return chunked(picks, n, [&](Q1Pick const *p, int c, int64_t) {
    q1_pick_kernel<<<dim3(blocks_for(per, 256), c), 256, 0, stream>>>(slots, p, x, g.dilE);
  });
}

cudaError_t q2(double2 *slots, Q2Inst const *inst, int64_t n, double2 const *q2m_,
               double2 const *peram, Geometry g, cudaStream_t stream) {
  int64_t const per = 16LL * g.dilE * g.dilE;
  return chunked(inst, n, [&](Q2Inst const *p, int c, int64_t) {
    q2_kernel<<<dim3(blocks_for(per, 256), c), 256, 0, stream>>>(slots, p, q2m_, peram, g);
  });
}

cudaError_t products(double2 *slots, ProdInst const *p, int64_t n, int32_t eds,
                     cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  size_t const smem = 2 * sizeof(double2) * eds * eds;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(product_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess) return e;
  }
  for (int64_t s = 0; s < n; s += 0x7fffffffLL) {
    int64_t const c = n - s < 0x7fffffffLL ? n - s : 0x7fffffffLL;
    product_kernel<<<static_cast<unsigned>(c), 256, smem, stream>>>(slots, p + s, eds);
  }
  return cudaGetLastError();
}

cudaError_t traces(double2 *values, TraceList const *lists, int32_t const *which,
                   int64_t n_which, int32_t const *shape_i, int32_t const *shape_j,
                   int64_t const *shape_off, double2 const *slots, int32_t eds,
                   cudaStream_t stream) {
  if (n_which == 0) return cudaSuccess;
  trace_kernel<<<static_cast<unsigned>(n_which), 256, 0, stream>>>(
      values, lists, which, shape_i, shape_j, shape_off, slots, eds);
  return cudaGetLastError();
}

cudaError_t terms(double2 *term_val, Term const *t, int64_t n, TraceList const *lists,
                  double2 const *values, uint16_t const *shape_mask,
                  int64_t const *shape_off, int32_t kahan, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  term_kernel<<<blocks_for(n, 128), 128, 0, stream>>>(term_val, t, n, lists, values,
                                                      shape_mask, shape_off, kahan);
  return cudaGetLastError();
}

cudaError_t divide(double2 *x, int64_t n, double d, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  divide_kernel<<<blocks_for(n, 256), 256, 0, stream>>>(x, n, d);
  return cudaGetLastError();
}

cudaError_t accumulate(double2 *running, int32_t const *seg_out, int64_t const *seg_off,
                       int64_t n_seg, int32_t const *idx, double2 const *term_val,
                       cudaStream_t stream) {
  if (n_seg == 0) return cudaSuccess;
  accumulate_kernel<<<blocks_for(n_seg, 128), 128, 0, stream>>>(running, seg_out, seg_off,
                                                               n_seg, idx, term_val);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace slaph

// ---------------------------------------------------------------- double-float
// Split-precision traces for the mixed path.  Matrices are converted once to
// double-float form (hi = fl32(x), lo = fl32(x - hi)), 16 bytes per complex
// like the FP64 layout; tr(L R) is then a compensated dot product on the FP32
// units (error-free products via FMA, Knuth two-sum accumulation, the cross
// terms hi*lo added to the compensation), summed in FP64 across the warp.
// GB300's FP32 units are ~60x faster than its FP64 units.
namespace slaph {
namespace dev {
namespace {

struct DfAcc {
  float s, c;
};
// acc += (xh + xl)(yh + yl), dropping xl*yl (relative 2^-48): error-free
// product by FMA, Knuth two-sum into s, all low-order parts into c.
__device__ __forceinline__ void df_mac(DfAcc &a, float xh, float xl, float yh, float yl) {
  float const p = xh * yh;
  float const e = fmaf(xh, yh, -p);
  float const s = a.s + p;
  float const bb = s - a.s;
  float const err = (a.s - (s - bb)) + (p - bb);
  a.s = s;
  a.c += err + e + fmaf(xh, yl, xl * yh);
}

// Warp sum of (s, c) pairs with error-free two-sums (FP32 units only).
__device__ __forceinline__ void df_warp_sum(DfAcc &a) {
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) {
    float const os = __shfl_down_sync(0xffffffffu, a.s, sh);
    float const oc = __shfl_down_sync(0xffffffffu, a.c, sh);
    float const s = a.s + os;
    float const bb = s - a.s;
    float const err = (a.s - (s - bb)) + (os - bb);
    a.s = s;
    a.c += oc + err;
  }
}

__global__ void __launch_bounds__(256) trace_df_kernel(double2 *values, TraceList const *lists,
                                                       int32_t const *which,
                                                       int32_t const *shape_i,
                                                       int32_t const *shape_j,
                                                       int64_t const *shape_off,
                                                       float4 const *slots_n,
                                                       float4 const *slots_t, int32_t eds) {
  TraceList const L = lists[which[blockIdx.x]];
  int64_t const off = shape_off[L.shape];
  int const n = static_cast<int>(shape_off[L.shape + 1] - off);
  int const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  int64_t const ms = static_cast<int64_t>(eds) * eds;
  for (int e = warp; e < n; e += blockDim.x / 32) {
    int const ia = shape_i[off + e], jb = shape_j[off + e];
    float4 const *A = slots_n + (static_cast<int64_t>(L.a_base) + ia) * ms;
    DfAcc ar{0.f, 0.f}, ai{0.f, 0.f};
    if (jb >= 0) {
      float4 const *B = slots_t + (static_cast<int64_t>(L.b_base) + jb) * ms;
      DfAcc br{0.f, 0.f}, bi{0.f, 0.f};  // second accumulator set (ILP)
      int64_t k = lane;
      for (; k + 32 < ms; k += 64) {
        float4 const x0 = A[k], y0 = B[k];
        float4 const x1 = A[k + 32], y1 = B[k + 32];
        df_mac(ar, x0.x, x0.y, y0.x, y0.y);
        df_mac(br, x1.x, x1.y, y1.x, y1.y);
        df_mac(ar, -x0.z, -x0.w, y0.z, y0.w);
        df_mac(br, -x1.z, -x1.w, y1.z, y1.w);
        df_mac(ai, x0.x, x0.y, y0.z, y0.w);
        df_mac(bi, x1.x, x1.y, y1.z, y1.w);
        df_mac(ai, x0.z, x0.w, y0.x, y0.y);
        df_mac(bi, x1.z, x1.w, y1.x, y1.y);
      }
      for (; k < ms; k += 32) {
        float4 const x = A[k], y = B[k];
        df_mac(ar, x.x, x.y, y.x, y.y);
        df_mac(ar, -x.z, -x.w, y.z, y.w);
        df_mac(ai, x.x, x.y, y.z, y.w);
        df_mac(ai, x.z, x.w, y.x, y.y);
      }
      df_mac(ar, br.s, br.c, 1.f, 0.f);
      df_mac(ai, bi.s, bi.c, 1.f, 0.f);
    } else {
      for (int i = lane; i < eds; i += 32) {
        float4 const x = A[i + static_cast<int64_t>(eds) * i];
        df_mac(ar, x.x, x.y, 1.f, 0.f);
        df_mac(ai, x.z, x.w, 1.f, 0.f);
      }
    }
    df_warp_sum(ar);
    df_warp_sum(ai);
    if (lane == 0)
      values[L.val_off + static_cast<int64_t>(e) * L.stride] =
          make_double2(static_cast<double>(ar.s) + static_cast<double>(ar.c),
                       static_cast<double>(ai.s) + static_cast<double>(ai.c));
  }
}

// Mixed path: C = A B in double-float arithmetic (operator*,
// src/DilutedFactor.cpp:40-41).  Both operands are staged in shared memory as
// stored (column-major): consecutive threads read consecutive rows of A and a
// broadcast element of B.  The result is written in both layouts, so products
// never pass through FP64.
__global__ void __launch_bounds__(256) product_df_kernel(float4 *slots_n, float4 *slots_t,
                                                         ProdInst const *p, int32_t eds) {
  extern __shared__ float4 sdf[];
  ProdInst const in = p[blockIdx.x];
  int64_t const ms = static_cast<int64_t>(eds) * eds;
  float4 *As = sdf, *Bs = sdf + ms;  // As[i + eds k] = A(i, k); Bs[k + eds j] = B(k, j)
  float4 const *A = slots_n + in.a * ms;
  float4 const *B = slots_n + in.b * ms;
  for (int k = threadIdx.x; k < ms; k += blockDim.x) {
    As[k] = A[k];
    Bs[k] = B[k];
  }
  __syncthreads();
  // Thread (i, c) computes the four entries (i, jb + c + u per), u = 0..3, of
  // each pass: one load of A(i, q) serves four multiply-adds, and the B loads
  // of a warp (one column per warp when eds >= 32) are broadcasts.
  int const per = blockDim.x / eds;
  int const i = threadIdx.x % eds, c = threadIdx.x / eds;
  if (c >= per) return;
  for (int jb = 0; jb < eds; jb += 4 * per) {
    DfAcc ar[4], ai[4];
    int jj[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      ar[u] = ai[u] = DfAcc{0.f, 0.f};
      jj[u] = min(jb + c + u * per, eds - 1);  // clamped: computed, not stored
    }
    for (int q = 0; q < eds; ++q) {
      float4 const x = As[i + eds * q];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float4 const y = Bs[q + eds * jj[u]];
        df_mac(ar[u], x.x, x.y, y.x, y.y);
        df_mac(ar[u], -x.z, -x.w, y.z, y.w);
        df_mac(ai[u], x.x, x.y, y.z, y.w);
        df_mac(ai[u], x.z, x.w, y.x, y.y);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      int const j = jb + c + u * per;
      if (j >= eds) break;
      float const rh = ar[u].s + ar[u].c, ih = ai[u].s + ai[u].c;
      float4 const f =
          make_float4(rh, ar[u].c - (rh - ar[u].s), ih, ai[u].c - (ih - ai[u].s));
      slots_n[in.c * ms + i + static_cast<int64_t>(eds) * j] = f;
      slots_t[in.c * ms + j + static_cast<int64_t>(eds) * i] = f;
    }
  }
}

}  // namespace

cudaError_t products_df(float4 *slots_n, float4 *slots_t, ProdInst const *p, int64_t n,
                        int32_t eds, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  if (eds < 1 || eds > 256) return cudaErrorInvalidValue;  // one row per thread of 256
  size_t const smem = 2 * sizeof(float4) * eds * eds;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(product_df_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess) return e;
  }
  for (int64_t s0 = 0; s0 < n; s0 += 0x7fffffffLL) {
    int64_t const c = n - s0 < 0x7fffffffLL ? n - s0 : 0x7fffffffLL;
    product_df_kernel<<<static_cast<unsigned>(c), 256, smem, stream>>>(slots_n, slots_t, p + s0,
                                                                        eds);
  }
  return cudaGetLastError();
}

cudaError_t traces_df(double2 *values, TraceList const *lists, int32_t const *which,
                      int64_t n_which, int32_t const *shape_i, int32_t const *shape_j,
                      int64_t const *shape_off, float4 const *slots_n, float4 const *slots_t,
                      int32_t eds, cudaStream_t stream) {
  if (n_which == 0) return cudaSuccess;
  trace_df_kernel<<<static_cast<unsigned>(n_which), 256, 0, stream>>>(
      values, lists, which, shape_i, shape_j, shape_off, slots_n, slots_t, eds);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace slaph

// ---------------------------------------------------------------- df factors
// Mixed path: the diluted-factor kernels above in double-float arithmetic.
// Inputs (VdaggerV, perambulators, noise) are converted once per
// configuration; the factors are written in both layouts for the products and
// traces.  Same formulas and reference lines as the FP64 kernels.
namespace slaph {
namespace dev {
namespace {

struct CDf {
  DfAcc r, i;
};
__device__ __forceinline__ CDf cdf_zero() { return CDf{{0.f, 0.f}, {0.f, 0.f}}; }
// acc += x * y
__device__ __forceinline__ void cdf_mac(CDf &a, float4 x, float4 y) {
  df_mac(a.r, x.x, x.y, y.x, y.y);
  df_mac(a.r, -x.z, -x.w, y.z, y.w);
  df_mac(a.i, x.x, x.y, y.z, y.w);
  df_mac(a.i, x.z, x.w, y.x, y.y);
}
// acc += conj(x) * y
__device__ __forceinline__ void cdf_macc(CDf &a, float4 x, float4 y) {
  df_mac(a.r, x.x, x.y, y.x, y.y);
  df_mac(a.r, x.z, x.w, y.z, y.w);
  df_mac(a.i, x.x, x.y, y.z, y.w);
  df_mac(a.i, -x.z, -x.w, y.x, y.y);
}
__device__ __forceinline__ float4 cdf_value(CDf const &a) {
  float const rh = a.r.s + a.r.c, ih = a.i.s + a.i.c;
  return make_float4(rh, a.r.c - (rh - a.r.s), ih, a.i.c - (ih - a.i.s));
}
// exact for the gamma values +-1, +-i
__device__ __forceinline__ float4 gamma_mul(double2 g, float4 v) {
  if (g.y == 0.0) return g.x > 0 ? v : make_float4(-v.x, -v.y, -v.z, -v.w);
  return g.y > 0 ? make_float4(-v.z, -v.w, v.x, v.y) : make_float4(v.z, v.w, -v.x, -v.y);
}
__device__ __forceinline__ float4 conj_df(float4 v) { return make_float4(v.x, v.y, -v.z, -v.w); }

__global__ void to_df_kernel(float4 *dst, double2 const *src, int64_t n) {
  int64_t const k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (k >= n) return;
  double2 const v = src[k];
  float const rh = static_cast<float>(v.x), ih = static_cast<float>(v.y);
  dst[k] = make_float4(rh, static_cast<float>(v.x - static_cast<double>(rh)), ih,
                       static_cast<float>(v.y - static_cast<double>(ih)));
}

__device__ __forceinline__ float4 const *vdv_block_df(float4 const *vdv, int code, int t,
                                                      Geometry const &g) {
  return vdv + (static_cast<int64_t>(code) * g.Lt + t) * g.nev * static_cast<int64_t>(g.nev);
}

// A thread takes the four Dirac indices d of one (v, e): they share the entries
// of VdaggerV (32^3x64 block pair: 1.5 -> 1.1 ms each for q0m and q1r).
__global__ void q0m_df_kernel(float4 *out, Q0MInst const *inst, float4 const *vdv,
                              float4 const *noise, Geometry g) {
  Q0MInst const in = inst[blockIdx.y];
  int const nev = g.nev, eds = 4 * g.dilE;
  int const k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nev * g.dilE) return;
  int const v = k % nev, e = k / nev;
  float4 const *m = vdv_block_df(vdv, in.vdv, in.t, g);
  float4 const *rho = noise + static_cast<int64_t>(in.r2) * g.Lt * 4 * nev;
  CDf acc[4] = {cdf_zero(), cdf_zero(), cdf_zero(), cdf_zero()};
  for (int w = e; w < nev; w += g.dilE) {
    float4 const x = m[v + static_cast<int64_t>(nev) * w];
    float4 const *rw = rho + 4 * (w + static_cast<int64_t>(nev) * in.t);
#pragma unroll
    for (int d = 0; d < 4; ++d) cdf_mac(acc[d], rw[d], x);
  }
  float4 *o = out + static_cast<int64_t>(blockIdx.y) * nev * eds + v;
#pragma unroll
  for (int d = 0; d < 4; ++d) o[static_cast<int64_t>(nev) * (e + g.dilE * d)] = cdf_value(acc[d]);
}

__global__ void q1r_df_kernel(float4 *out, Q1RInst const *inst, float4 const *vdv,
                              float4 const *noise, Geometry g) {
  Q1RInst const in = inst[blockIdx.y];
  int const nev = g.nev, eds = 4 * g.dilE;
  int const k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nev * g.dilE) return;
  int const e = k % g.dilE, j = k / g.dilE;
  float4 const *m = vdv_block_df(vdv, in.vdv, in.t, g);
  float4 const *rho = noise + static_cast<int64_t>(in.r1) * g.Lt * 4 * nev;
  CDf acc[4] = {cdf_zero(), cdf_zero(), cdf_zero(), cdf_zero()};
  for (int v = e; v < nev; v += g.dilE) {
    float4 const x = m[v + static_cast<int64_t>(nev) * j];
    float4 const *rv = rho + 4 * (v + static_cast<int64_t>(nev) * in.t);
#pragma unroll
    for (int d = 0; d < 4; ++d) cdf_macc(acc[d], rv[d], x);
  }
  float4 *o = out + static_cast<int64_t>(blockIdx.y) * nev * eds + e + static_cast<int64_t>(eds) * j;
#pragma unroll
  for (int d = 0; d < 4; ++d) o[g.dilE * d] = cdf_value(acc[d]);
}

__device__ __forceinline__ void store_factor_df(float4 *sn, float4 *st, int slot, int k, int eds,
                                                float4 v) {
  int64_t const ms = static_cast<int64_t>(eds) * eds;
  int const i = k % eds, j = k / eds;
  sn[slot * ms + k] = v;
  st[slot * ms + j + static_cast<int64_t>(eds) * i] = v;
}

__global__ void q0_df_kernel(float4 *sn, float4 *st, Q0Inst const *inst, float4 const *q0m,
                             float4 const *noise, unsigned int *slot_bits, Geometry g) {
  Q0Inst const in = inst[blockIdx.y];
  int const nev = g.nev, dilE = g.dilE, eds = 4 * dilE;
  int const k = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned int mx = 0;
  if (k < eds * eds) {
    int const a = k % eds, b = k / eds;
    int const d = b / dilE;
    int const gr = c_gamma_row[in.gamma][d];
    CDf acc = cdf_zero();
    if (a / dilE == gr) {
      int const e1 = a % dilE;
      float4 const *M = q0m + static_cast<int64_t>(in.m) * nev * eds;
      float4 const *rho = noise + static_cast<int64_t>(in.r1) * g.Lt * 4 * nev;
      double2 const val = c_gamma_val[in.gamma][d];
      for (int v = e1; v < nev; v += dilE)
        cdf_mac(acc, gamma_mul(val, M[v + static_cast<int64_t>(nev) * b]),
                conj_df(rho[gr + 4 * (v + static_cast<int64_t>(nev) * in.t)]));
    }
    float4 const f = cdf_value(acc);
    mx = max(__float_as_uint(f.x) & 0x7FFFFFFFu, __float_as_uint(f.z) & 0x7FFFFFFFu);
    store_factor_df(sn, st, in.slot, k, eds, f);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (threadIdx.x % 32 == 0 && mx != 0) atomicMax(slot_bits + in.slot, mx);
}

int blocks256(int64_t n) { return static_cast<int>((n + 255) / 256); }

}  // namespace

cudaError_t to_df(float4 *dst, double2 const *src, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  to_df_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(dst, src, n);
  return cudaGetLastError();
}

cudaError_t factors_df(float4 *sn, float4 *st, float4 *q0m_buf, float4 *q1r_buf,
                       Q0MInst const *q0m_i, int64_t n_q0m, Q1RInst const *q1r_i, int64_t n_q1r,
                       Q0Inst const *q0_i, int64_t n_q0, float4 const *vdv, float4 const *noise,
                       unsigned int *slot_bits, Geometry g, cudaStream_t stream) {
  int const eds = 4 * g.dilE;
  int64_t const per_m = static_cast<int64_t>(g.nev) * eds;
  int64_t const per_f = static_cast<int64_t>(eds) * eds;
  cudaError_t e;
  e = chunked(q0m_i, n_q0m, [&](Q0MInst const *p, int c, int64_t s) {
    q0m_df_kernel<<<dim3(blocks256(per_m / 4), c), 256, 0, stream>>>(q0m_buf + s * per_m, p, vdv,
                                                                 noise, g);
  });
  if (e != cudaSuccess) return e;
  e = chunked(q1r_i, n_q1r, [&](Q1RInst const *p, int c, int64_t s) {
    q1r_df_kernel<<<dim3(blocks256(per_m / 4), c), 256, 0, stream>>>(q1r_buf + s * per_m, p, vdv,
                                                                 noise, g);
  });
  if (e != cudaSuccess) return e;
  return chunked(q0_i, n_q0, [&](Q0Inst const *p, int c, int64_t) {
    q0_df_kernel<<<dim3(blocks256(per_f), c), 256, 0, stream>>>(sn, st, p, q0m_buf, noise, slot_bits, g);
  });
}

}  // namespace dev
}  // namespace slaph
