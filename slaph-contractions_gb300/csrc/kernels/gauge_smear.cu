// HYP smearing of the spatial gauge links (GaugeField::smearing_hyp,
// src/GaugeField.cpp:322-427), FP64, every timeslice of a chunk at once.
//
// One iteration is two launches:
//   inner: one thread per (timeslice, site, direction, perpendicular n) builds
//          the decorated link  P(U(s,d) (1 - a2) + (a2 / 2) staple_p)  where
//          staple_p is the up and down staple of U in direction p = get_dirs(d)[n]
//          (:336-376), stored at slot d + 3 n;
//   outer: one thread per (timeslice, site, direction) sums the staples of the
//          decorated links in both other directions, each taken from the slot
//          decor(., plane) of the plane that excludes it (:380-416), and
//          replaces U(s,d) by P(U(s,d) (1 - a1) + (a1 / 4) outer).
// Only a thread's own link is read from U in the outer launch, so it updates U
// in place.  P is proj_to_su3_imp (:203-210): M (M^H M)^(-1/2) scaled by the
// principal cube root of 1/det (proj_su3 below).
//
// Bound by FP64 issue (two multiply-adds per cycle and SM): about 1080
// operations per decorated link and 1500 per outer link.  24^3x48, three
// iterations: 134 ms with Jacobi eigen-decompositions of M^H M and FP64
// transcendentals, 41 ms with the closed form.
//
// Sites and neighbours follow GaugeField::init (src/GaugeField.cpp:39-98) on a
// cubic lattice: s = (x0 L + x1) L + x2, direction d steps x_d periodically.
// Links: [site][dir][a + 3 b] (column-major 3x3), 9 complex per link.
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.cuh"

namespace slaph {
namespace dev {
namespace {

struct M3 {
  double2 e[9];  // (a, b) at a + 3 b
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double cnorm(double2 a) { return a.x * a.x + a.y * a.y; }

// acc + a b, acc + conj(a) b, acc + a conj(b)
__device__ __forceinline__ double2 cmac(double2 acc, double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, fma(-a.y, b.y, acc.x)), fma(a.x, b.y, fma(a.y, b.x, acc.y)));
}
__device__ __forceinline__ double2 cmac_hn(double2 acc, double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, fma(a.y, b.y, acc.x)), fma(a.x, b.y, fma(-a.y, b.x, acc.y)));
}
__device__ __forceinline__ double2 cmac_nh(double2 acc, double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, fma(a.y, b.y, acc.x)), fma(a.y, b.x, fma(-a.x, b.y, acc.y)));
}
// acc - a b
__device__ __forceinline__ double2 cnmac(double2 acc, double2 a, double2 b) {
  return make_double2(fma(-a.x, b.x, fma(a.y, b.y, acc.x)), fma(-a.x, b.y, fma(-a.y, b.x, acc.y)));
}
__device__ __forceinline__ double2 det3(M3 const &m) {
  double2 const c0 = cnmac(cmul(m.e[4], m.e[8]), m.e[7], m.e[5]);
  double2 const c1 = cnmac(cmul(m.e[1], m.e[8]), m.e[7], m.e[2]);
  double2 const c2 = cnmac(cmul(m.e[1], m.e[5]), m.e[4], m.e[2]);
  return cmac(cnmac(cmul(m.e[0], c0), m.e[3], c1), m.e[6], c2);
}

__device__ __forceinline__ M3 load(double2 const *p) {
  M3 m;
#pragma unroll
  for (int i = 0; i < 9; ++i) m.e[i] = p[i];
  return m;
}
__device__ __forceinline__ void store(double2 *p, M3 const &m) {
#pragma unroll
  for (int i = 0; i < 9; ++i) p[i] = m.e[i];
}

// x y, x^H y, x y^H
__device__ __forceinline__ M3 mul(M3 const &x, M3 const &y) {
  M3 r;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b)
      r.e[a + 3 * b] = cmac(cmac(cmul(x.e[a], y.e[3 * b]), x.e[a + 3], y.e[1 + 3 * b]),
                            x.e[a + 6], y.e[2 + 3 * b]);
  return r;
}
__device__ __forceinline__ M3 mul_hn(M3 const &x, M3 const &y) {
  M3 r;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b)
      r.e[a + 3 * b] = cmac_hn(cmac_hn(cmul(cconj(x.e[3 * a]), y.e[3 * b]), x.e[1 + 3 * a],
                                       y.e[1 + 3 * b]),
                               x.e[2 + 3 * a], y.e[2 + 3 * b]);
  return r;
}
__device__ __forceinline__ M3 mul_nh(M3 const &x, M3 const &y) {
  M3 r;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b)
      r.e[a + 3 * b] = cmac_nh(cmac_nh(cmul(x.e[a], cconj(y.e[b])), x.e[a + 3], y.e[b + 3]),
                               x.e[a + 6], y.e[b + 6]);
  return r;
}

// cof(X): X^(-1) = cof(X)^T / det X.
__device__ __forceinline__ M3 cofactors(M3 const &x) {
  M3 r;
#pragma unroll
  for (int b = 0; b < 3; ++b)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      int const r1 = (a + 1) % 3, r2 = (a + 2) % 3, s1 = 3 * ((b + 1) % 3), s2 = 3 * ((b + 2) % 3);
      r.e[a + 3 * b] = cnmac(cmul(x.e[r1 + s1], x.e[r2 + s2]), x.e[r1 + s2], x.e[r2 + s1]);
    }
  return r;
}

// proj_to_su3_imp (src/GaugeField.cpp:203-210) for a matrix of any condition and
// scale: Newton's iteration on the polar decomposition, X -> (g X + X^(-H) / g) / 2 with
// g^2 = |X^(-1)| / |X| (Higham, SIAM J. Sci. Stat. Comput. 7 (1986) 1160), from X = M
// scaled to entries of order one; at most nine steps for singular values 1e16 apart,
// the last of them with g = 1 to rounding.  Largest error for singular values 1, s, s
// (100 random matrices each; from the eigenvectors of M^H M in brackets): 3e-16 at s =
// 0.1 (3e-15), 2e-14 at 1e-2 (3e-13), 2e-10 at 1e-4 (3e-9), 2e-8 at 1e-5 (7e-7).
__device__ __noinline__ M3 polar_su3(M3 x) {
  double top = 0;
  for (int i = 0; i < 9; ++i) top = fmax(top, fmax(fabs(x.e[i].x), fabs(x.e[i].y)));
  int e;
  frexp(top, &e);
  for (int i = 0; i < 9; ++i)
    x.e[i] = make_double2(scalbn(x.e[i].x, -e), scalbn(x.e[i].y, -e));
  for (int k = 0; k < 16; ++k) {
    M3 const cf = cofactors(x);
    double nx = 0, nc = 0;
    for (int i = 0; i < 9; ++i) {
      nx += cnorm(x.e[i]);
      nc += cnorm(cf.e[i]);
    }
    double2 const d = cmac(cmac(cmul(x.e[0], cf.e[0]), x.e[1], cf.e[1]), x.e[2], cf.e[2]);
    double const n2 = cnorm(d);
    double const g = sqrt(sqrt(nc / n2 / nx));
    double const h = 0.5 / (g * n2);
    double2 const hd = make_double2(d.x * h, d.y * h);  // 1 / (2 g conj(det X))
    double moved = 0;
    for (int i = 0; i < 9; ++i) {
      double2 const t = cmul(hd, cconj(cf.e[i]));
      double2 const y = make_double2(fma(0.5 * g, x.e[i].x, t.x), fma(0.5 * g, x.e[i].y, t.y));
      moved += cnorm(make_double2(y.x - x.e[i].x, y.y - x.e[i].y));
      x.e[i] = y;
    }
    if (!(moved > 1e-18)) break;  // quadratic: the next step would move by 1e-18 / 2
  }
  double2 const d = det3(x);
  double sn, cs;
  sincos(-atan2(d.y, d.x) / 3.0, &sn, &cs);
  for (int i = 0; i < 9; ++i) x.e[i] = cmul(x.e[i], make_double2(cs, sn));
  return x;
}

// proj_to_su3_imp (src/GaugeField.cpp:203-210) in closed form.  With A = M^H M
// and u, v, w the elementary symmetric functions of the singular values of M
// (the square roots of A's eigenvalues), the Cayley-Hamilton theorem gives
//   A^(-1/2) = f0 + f1 A + f2 A^2,  d = w (u v - w),
//   f0 = (u v^2 - w (u^2 + v)) / d, f1 = (2 u v - u^3 - w) / d, f2 = u / d
// (Hasenfratz, Hoffmann, Schaefer, JHEP 05 (2007) 029); d is a product of sums
// of singular values, so nothing cancels where they approach one another.  Where two
// of them are small beside the third, v cancels, the quartic's two largest roots meet
// and the Newton steps below stop early: from c2 = 0.1 c1^2 down (singular values 1, 0.35,
// 0.35 or 1, 0.4, 0; 1/3 for a multiple of a unitary matrix) polar_su3 takes over, as
// it does where powers of the links' scale would leave the range of FP64.  300 matrices
// each for 1476 pairs of smaller singular values (0.3 to 1, and that down to 1e-9 of it):
// the largest error is nowhere above that from eigenvectors; the closed form alone is
// three times above it at c2 = 0.02 c1^2.
// w = |det M|; u is the largest root of (u^2 - tr A)^2 - 8 w u - 4 c2 (c2 the
// sum of A's principal minors), found by Newton's method from above, where the
// quartic is convex: FP32 steps from sqrt(3 tr A), then FP64 steps until the
// next correction is negligible; v = (u^2 - tr A) / 2.  The determinant of
// M A^(-1/2) is det M / w: its principal root y = (det M / w)^(-1/3) comes from
// FP32 and two FP64 Newton steps y (4 - y^3 z) / 3.  One Newton step of the
// polar decomposition, X -> (X + X^(-H)) / 2, ends it: whatever error of f0, f1,
// f2 is left enters squared, and the result is more accurate than one from
// A's eigenvectors (1.2e-16 rms against 3.7e-16 on blends with singular values
// 0.7 .. 1; 8.8e-16 without the step).
__device__ M3 proj_su3(M3 const &m) {
  // A: diagonal a0, a1, a2 and upper entries p = A01, q = A02, r = A12
  double a[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    a[i] = cnorm(m.e[3 * i]);
#pragma unroll
    for (int k = 1; k < 3; ++k)
      a[i] = fma(m.e[k + 3 * i].x, m.e[k + 3 * i].x,
                 fma(m.e[k + 3 * i].y, m.e[k + 3 * i].y, a[i]));
  }
  auto dot = [&](int i, int j) {
    return cmac_hn(cmac_hn(cmul(cconj(m.e[3 * i]), m.e[3 * j]), m.e[1 + 3 * i], m.e[1 + 3 * j]),
                   m.e[2 + 3 * i], m.e[2 + 3 * j]);
  };
  double2 const p = dot(0, 1), q = dot(0, 2), r = dot(1, 2);
  double const np = cnorm(p), nq = cnorm(q), nr = cnorm(r);
  double const c1 = a[0] + a[1] + a[2];
  double const c2 = (fma(a[0], a[1], -np) + fma(a[0], a[2], -nq)) + fma(a[1], a[2], -nr);
  // c2 / c1^2 in FP32, the scale by the exponent of c1 (2^-64 .. 2^64): no FP64 operation
  double const is = rsqrt(c1), is2 = is * is;
  float const t2 = static_cast<float>(4 * c2 * is2 * is2);
  unsigned int const scale = static_cast<unsigned int>(__double2hiint(c1)) - ((1023u - 64u) << 20);
  if (!(t2 > 0.4f) || scale >= 128u << 20) return polar_su3(m);
  double2 const det = det3(m);
  double const d2 = cnorm(det);
  double const iw = rsqrt(d2);
  double const w = d2 * iw;
  // in units of sqrt(tr A) while in FP32
  float const tw = static_cast<float>(8 * w * is2 * is);
  float x0 = 1.7320508f;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    float const g = x0 * x0 - 1.f, dp = 4.f * x0 * g - tw;
    float const step = (g * g - tw * x0 - t2) / dp;
    if (step > 0.f) x0 -= step;  // from above; rounding ends the descent
  }
  double u = static_cast<double>(x0) * (c1 * is);
  for (int k = 0; k < 30; ++k) {
    double const g = fma(u, u, -c1);
    double const pu = fma(g, g, -fma(8 * w, u, 4 * c2));
    double const step = pu / fma(4 * u, g, -8 * w);
    u -= step;
    if (!(fabs(step) > 1e-5 * u)) break;  // quadratic: the next step is about 1e-10
  }
  double const v = 0.5 * fma(u, u, -c1);
  double const uv = u * v;
  double const id = iw / (uv - w);
  double const f2 = u * id;
  double const f1 = (fma(2.0, uv, -w) - u * u * u) * id;
  double const f0 = fma(uv, v, -w * fma(u, u, v)) * id;
  // B = f0 + f1 A + f2 A^2 (Hermitian, same storage as A)
  double const b0 = fma(f2, fma(a[0], a[0], np + nq), fma(f1, a[0], f0));
  double const b1 = fma(f2, fma(a[1], a[1], np + nr), fma(f1, a[1], f0));
  double const b2 = fma(f2, fma(a[2], a[2], nq + nr), fma(f1, a[2], f0));
  // (A^2)01 = A01 (a0 + a1) + A02 conj(A12) and so on
  auto off = [&](double2 z, double s, double2 zz) {
    double const c = fma(f2, s, f1);
    return make_double2(fma(c, z.x, f2 * zz.x), fma(c, z.y, f2 * zz.y));
  };
  double2 const zero = make_double2(0, 0);
  double2 const bp = off(p, a[0] + a[1], cmac_nh(zero, q, r));
  double2 const bq = off(q, a[0] + a[2], cmul(p, r));
  double2 const br = off(r, a[1] + a[2], cmac_hn(zero, p, q));
  // y = (det / w)^(-1/3)
  double2 const z = make_double2(det.x * iw, det.y * iw);
  float sf, cf;
  sincosf(-atan2f(static_cast<float>(z.y), static_cast<float>(z.x)) / 3.f, &sf, &cf);
  double2 y = make_double2(static_cast<double>(cf), static_cast<double>(sf));
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    double2 const y3z = cmul(cmul(cmul(y, y), y), z);
    y = cmul(y, make_double2((4.0 - y3z.x) * (1.0 / 3.0), -y3z.y * (1.0 / 3.0)));
  }
  M3 x;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double2 const m0 = cmul(m.e[i], y), m1 = cmul(m.e[i + 3], y), m2 = cmul(m.e[i + 6], y);
    auto real = [](double2 acc, double2 t, double s) {
      return make_double2(fma(t.x, s, acc.x), fma(t.y, s, acc.y));
    };
    // columns of B: (b0, conj p, conj q), (p, b1, conj r), (q, r, b2)
    x.e[i] = cmac_nh(cmac_nh(make_double2(m0.x * b0, m0.y * b0), m1, bp), m2, bq);
    x.e[i + 3] = cmac_nh(real(cmul(m0, bp), m1, b1), m2, br);
    x.e[i + 6] = real(cmac(cmul(m0, bq), m1, br), m2, b2);
  }
  // (X + conj(cof X) / conj(det X)) / 2
  M3 const cf3 = cofactors(x);
  double2 const dx =
      cmac(cmac(cmul(x.e[0], cf3.e[0]), x.e[1], cf3.e[1]), x.e[2], cf3.e[2]);
  double const h = 0.5 / cnorm(dx);
  double2 const hd = make_double2(dx.x * h, dx.y * h);  // 1 / (2 conj(det X))
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    double2 const t = cmul(hd, cconj(cf3.e[i]));
    x.e[i] = make_double2(fma(0.5, x.e[i].x, t.x), fma(0.5, x.e[i].y, t.y));
  }
  return x;
}

__device__ __forceinline__ int64_t step(int64_t s, int dir, int L, int delta) {
  int64_t const stride = dir == 0 ? static_cast<int64_t>(L) * L : (dir == 1 ? L : 1);
  int const c = static_cast<int>((s / stride) % L);
  int const nc = (c + delta + L) % L;
  return s + (nc - c) * stride;
}

__device__ __forceinline__ double2 const *link(double2 const *U, int64_t s, int dir) {
  return U + (3 * s + dir) * 9;
}

// Decorated links of one chunk: dec[(t V3 + s) 6 + d + 3 n].
__global__ void hyp_inner_kernel(double2 *dec, double2 const *U, int32_t L, int64_t V3,
                                 int64_t n_items, double alpha2) {
  int64_t const k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (k >= n_items) return;
  int64_t const ts = k / 6;  // t V3 + s
  int const slot = static_cast<int>(k % 6);
  int const dir = slot % 3, n = slot / 3;
  int const perp = n == 0 ? (dir == 0 ? 1 : 0) : (dir == 2 ? 1 : 2);
  int64_t const t = ts / V3, s = ts % V3;
  double2 const *Ut = U + t * V3 * 27;
  int64_t const s_up = step(s, perp, L, 1), s_dir = step(s, dir, L, 1);
  int64_t const s_dn = step(s, perp, L, -1), s_dn_dir = step(s_dn, dir, L, 1);
  M3 st = mul(load(link(Ut, s, perp)), mul_nh(load(link(Ut, s_up, dir)), load(link(Ut, s_dir, perp))));
  M3 const dn = mul_hn(load(link(Ut, s_dn, perp)),
                       mul(load(link(Ut, s_dn, dir)), load(link(Ut, s_dn_dir, perp))));
  M3 const u = load(link(Ut, s, dir));
  double const w = 1 - alpha2, a = alpha2 / 2.;
#pragma unroll
  for (int i = 0; i < 9; ++i)
    st.e[i] = make_double2(u.e[i].x * w + (st.e[i].x + dn.e[i].x) * a,
                           u.e[i].y * w + (st.e[i].y + dn.e[i].y) * a);
  store(dec + k * 9, proj_su3(st));
}

// decor (src/GaugeField.cpp:170-190): slot of the link in direction d that
// was smeared with the third direction `plane`.
__device__ __forceinline__ int decor(int d, int plane) {
  if (d == 0) return plane == 1 ? 0 : 3;
  if (d == 1) return plane == 0 ? 1 : 4;
  return plane == 0 ? 2 : 5;
}

__global__ void hyp_outer_kernel(double2 *U, double2 const *dec, int32_t L, int64_t V3,
                                 int64_t n_items, double alpha1) {
  int64_t const k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (k >= n_items) return;
  int64_t const ts = k / 3;
  int const dir = static_cast<int>(k % 3);
  int64_t const t = ts / V3, s = ts % V3;
  double2 const *Dt = dec + t * V3 * 54;
  M3 outer;
#pragma unroll
  for (int i = 0; i < 9; ++i) outer.e[i] = make_double2(0, 0);
#pragma unroll 1  // (unrolled: 244 registers, half the warps per SM)
  for (int nd = 0; nd < 3; ++nd) {
    if (nd == dir) continue;
    int const plane = 3 - dir - nd;
    int const a = decor(nd, plane), b = decor(dir, plane);
    int64_t const s_up = step(s, nd, L, 1), s_dir = step(s, dir, L, 1);
    int64_t const s_dn = step(s, nd, L, -1), s_dn_dir = step(s_dn, dir, L, 1);
    M3 const up = mul(load(Dt + (6 * s + a) * 9),
                      mul_nh(load(Dt + (6 * s_up + b) * 9), load(Dt + (6 * s_dir + a) * 9)));
    M3 const dn = mul_hn(load(Dt + (6 * s_dn + a) * 9),
                         mul(load(Dt + (6 * s_dn + b) * 9), load(Dt + (6 * s_dn_dir + a) * 9)));
#pragma unroll
    for (int i = 0; i < 9; ++i) outer.e[i] = cadd(outer.e[i], cadd(up.e[i], dn.e[i]));
  }
  double2 *u = U + (t * V3 * 3 + 3 * s + dir) * 9;
  M3 const m = load(u);
  double const w = 1 - alpha1, c = alpha1 / 4.;
#pragma unroll
  for (int i = 0; i < 9; ++i)
    outer.e[i] = make_double2(m.e[i].x * w + outer.e[i].x * c, m.e[i].y * w + outer.e[i].y * c);
  store(u, proj_su3(outer));
}

inline unsigned blocks_of(int64_t n, int threads) {
  return static_cast<unsigned>((n + threads - 1) / threads);
}

}  // namespace

int64_t hyp_scratch_doubles_per_timeslice(int32_t L) {
  return static_cast<int64_t>(L) * L * L * 6 * 9 * 2;
}

cudaError_t hyp_smear(double2 *U, double2 *dec, int32_t L, int32_t n_t, double alpha1,
                      double alpha2, cudaStream_t stream) {
  if (L < 1 || n_t < 1) return cudaErrorInvalidValue;
  int64_t const V3 = static_cast<int64_t>(L) * L * L;
  int64_t const n_inner = n_t * V3 * 6, n_outer = n_t * V3 * 3;
  hyp_inner_kernel<<<blocks_of(n_inner, 128), 128, 0, stream>>>(dec, U, L, V3, n_inner, alpha2);
  cudaError_t const e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  hyp_outer_kernel<<<blocks_of(n_outer, 128), 128, 0, stream>>>(U, dec, L, V3, n_outer, alpha1);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace slaph
