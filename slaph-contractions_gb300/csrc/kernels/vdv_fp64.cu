// FP64 VdaggerV by momentum families (vdv_families.hpp).
//
// OperatorFactory::build_vdaggerv, src/OperatorFactory.cpp:292-300.  GB300 has
// two FP64 multiply-adds per cycle and SM (1.25 TFLOP/s), so the kernel is
// bound by the number of multiply-adds and by how evenly they spread over the
// SMs; loads and shared memory are idle beside them.  Hence:
//
// * a family's plane sums without a phase are Hermitian: only entries i <= j
//   are computed, and a phase family serves up to three operators per pass;
// * a CTA takes a tile of (i, j) of 32 x 32 entries, two by two per thread (or
//   16 x 16, one per thread, where 32-wide tiles are too few for the chip), and
//   only the threads of wanted entries (i <= j, i, j < nev) run the
//   multiply-adds, packed into whole warps (the warp numbering is rotated per
//   CTA, so that the warps left over spread over the SM's four partitions);
// * the planes of a tile are split over a cluster of up to 8 CTAs until the
//   launch has 12 CTAs per SM; the partial sums meet in distributed shared
//   memory in a fixed order, without scratch memory.
//
// Measured against the 64 x 64 tile per (operator, timeslice) over the whole
// lattice that it replaces (all entries, phase applied while staging): 24^3,
// Nev 120, one momentum and timeslice 172 -> 2.75 ms (4 CTAs -> the chip);
// 14^3x24, Nev 51, three momenta 34.3 -> 7.4 ms; 24^3x48, Nev 64, three momenta
// 173 -> 101 ms (1.13 TFLOP/s of all entries -> 0.97 of the wanted half).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "kernels.cuh"
#include "vdv_families.hpp"

namespace slaph {
namespace dev {

namespace {

constexpr int kK = 16;        // lattice entries per step
constexpr int kThr = 256;     // 16 x 16 threads, kB x kB entries each
constexpr int kMaxFam = 16;   // families per launch
static_assert(kVdvFp64Ops == 3, "kernel instances");

struct FamilyArgs {
  VdvFamily f[kMaxFam];
};

// conj(a) b added to acc.
__device__ __forceinline__ void mac(double2 &acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, fma(a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(-a.y, b.x, acc.y));
}

// cos and sin of 2 pi n / d.
__device__ __forceinline__ void unit(int64_t n, int32_t d, double *c, double *s) {
  sincospi(2.0 * static_cast<double>(n % d) / static_cast<double>(d), s, c);
}

struct Planes {
  VdvFamily const &f;
  int32_t Lx, Ly, Lz;
  int32_t per;  // entries per plane
  __device__ Planes(VdvFamily const &fam, Geometry const &g)
      : f(fam), Lx(g.Lx), Ly(g.Ly), Lz(g.Lz) {
    int32_t const sites = f.axis == 0   ? Ly * Lz
                          : f.axis == 1 ? Lx * Lz
                          : f.axis == 2 ? Lx * Ly
                                        : Lx * Ly * Lz;
    per = 3 * sites;
  }
  // Site index and coordinates of site q of plane h.
  __device__ __forceinline__ int64_t site(int32_t h, int32_t q, int32_t (&x)[3]) const {
    if (f.axis == 3) {
      x[0] = q / (Ly * Lz);
      x[1] = q / Lz % Ly;
      x[2] = q % Lz;
      return q;
    }
    int32_t const lv = f.axis == 2 ? Ly : Lz;
    int32_t const u = q / lv, v = q - u * lv;
    int64_t const L = f.n_planes;
    int64_t m = (h - static_cast<int64_t>(f.sh_u) * u - static_cast<int64_t>(f.sh_v) * v) % L;
    if (m < 0) m += L;
    if (f.sgn < 0 && m > 0) m = L - m;
    int32_t const xa = static_cast<int32_t>(m);
    x[0] = f.axis == 0 ? xa : u;
    x[1] = f.axis == 1 ? xa : f.axis == 0 ? u : v;
    x[2] = f.axis == 2 ? xa : v;
    return (static_cast<int64_t>(x[0]) * Ly + x[1]) * Lz + x[2];
  }
};

// kB: entries per thread and side.  kHerm: plane sums of V with itself, i <= j.
// kOps: operators of the family.  kW: B = W, a displaced copy of V_t (one
// operator and timeslice per launch).
template <int kB, bool kHerm, int kOps, bool kW>
__global__ void __launch_bounds__(kThr, kHerm && kOps > 2 ? 1 : 2)
    vdv_family_kernel(double2 *vdv, double2 const *V, double2 const *W,
                      const __grid_constant__ FamilyArgs args, int32_t const *op_ids, int32_t t0,
                      int32_t v_t0, int32_t split, Geometry g) {
  namespace cg = cooperative_groups;
  constexpr int kSums = kHerm ? 4 : 2;  // doubles per entry and operator
  constexpr int kT = 16 * kB;           // entries (i or j) per tile side
  constexpr int kE = kB * kB;           // entries per thread
  constexpr int kLd = kT + 1;           // rows of a staged step, padded against bank conflicts
  // Staged operands of a step; after the loop the partial sums of one
  // operator, [kE entries x kSums][thread].
  __shared__ __align__(16) double smem[kE * kSums * kThr > 4 * kK * kLd ? kE * kSums * kThr
                                                                        : 4 * kK * kLd];
  __shared__ double2 phase[2][kK];
  __shared__ double2 turn[kOps];
  double2(*As)[kLd] = reinterpret_cast<double2(*)[kLd]>(smem);
  double2(*Bs)[kLd] = As + kK;

  VdvFamily const &f = args.f[blockIdx.y];
  Planes const pl(f, g);
  int const nev = g.nev;
  int const rank = static_cast<int>(blockIdx.x % split);
  int tile = static_cast<int>(blockIdx.x / split);
  int const nt = (nev + kT - 1) / kT;
  int ti, tj;
  if (kHerm) {  // tile (ti <= tj) at tj (tj + 1) / 2 + ti
    tj = 0;
    while ((tj + 1) * (tj + 2) / 2 <= tile) ++tj;
    ti = tile - tj * (tj + 1) / 2;
  } else {
    ti = tile % nt;
    tj = tile / nt;
  }
  int const i0 = ti * kT, j0 = tj * kT;
  bool const diag = kHerm && ti == tj;
  int const t = t0 + blockIdx.z;
  int const tid = threadIdx.x;
  double2 const *Vt = V + static_cast<int64_t>(t - v_t0) * nev * g.dim_row;
  double2 const *Bt = kW ? W : Vt;
  bool const has_phase = !kHerm && (f.w[0] != 0 || f.w[1] != 0 || f.w[2] != 0);

  // The block of entries of this thread among the wanted ones.
  int const nbi = (min(kT, nev - i0) + kB - 1) / kB, nbj = (min(kT, nev - j0) + kB - 1) / kB;
  int const n_act = diag ? nbi * (nbi + 1) / 2 : nbi * nbj;
  int const rot = static_cast<int>((blockIdx.x + 3 * blockIdx.y + 5 * blockIdx.z) % (kThr / 32));
  int const blk = ((tid / 32 + rot) % (kThr / 32)) * 32 + tid % 32;
  bool const warp_on = (blk & ~31) < n_act;
  int bi = 0, bj = 0;
  if (blk < n_act) {
    if (diag) {
      while ((bj + 1) * (bj + 2) / 2 <= blk) ++bj;
      bi = blk - bj * (bj + 1) / 2;
    } else {
      bi = blk % nbi;
      bj = blk / nbi;
    }
  }

  double2 acc[kE];
  double sum[kOps][kE][kSums];
#pragma unroll
  for (int e = 0; e < kE; ++e) {
    acc[e] = make_double2(0, 0);
#pragma unroll
    for (int o = 0; o < kOps; ++o)
#pragma unroll
      for (int s = 0; s < kSums; ++s) sum[o][e][s] = 0;
  }

  int64_t const spp = (pl.per + kK - 1) / kK;  // steps per plane
  int64_t const total = spp * f.n_planes;
  int64_t const s0 = total * rank / split, s1 = total * (rank + 1) / split;
  int const kk = tid % kK, row = tid / kK;  // this thread stages rows row, row + 16
  double2 ra[kB], rb[kB];
  // Global loads of step s into registers; the phases of its entries.
  auto fetch = [&](int64_t s) {
    int32_t const h = static_cast<int32_t>(s / spp);
    int32_t const k = static_cast<int32_t>(s - h * spp) * kK + kk;
    bool const in = k < pl.per;
    int32_t x[3];
    int64_t at = 0;
    if (in) at = 3 * pl.site(h, k / 3, x) + k % 3;
#pragma unroll
    for (int q = 0; q < kB; ++q) {
      int const i = i0 + row + 16 * q, j = j0 + row + 16 * q;
      ra[q] = in && i < nev ? Vt[static_cast<int64_t>(i) * g.dim_row + at] : make_double2(0, 0);
      if (!diag)
        rb[q] = in && j < nev ? Bt[static_cast<int64_t>(j) * g.dim_row + at] : make_double2(0, 0);
    }
    if (has_phase && tid < kK) {
      double c = 1, sn = 0;
      if (in) {
        double const a =
            static_cast<double>(static_cast<int64_t>(f.w[0]) * x[0] % g.Lx) / g.Lx +
            static_cast<double>(static_cast<int64_t>(f.w[1]) * x[1] % g.Ly) / g.Ly +
            static_cast<double>(static_cast<int64_t>(f.w[2]) * x[2] % g.Lz) / g.Lz;
        sincospi(2.0 * a, &sn, &c);
      }
      phase[s & 1][kk] = make_double2(c, -sn);
    }
  };
  if (s0 < s1) fetch(s0);
  for (int64_t s = s0; s < s1; ++s) {
    __syncthreads();  // the previous step's operands are consumed, phase[s & 1] is written
#pragma unroll
    for (int q = 0; q < kB; ++q) {
      As[kk][row + 16 * q] = ra[q];
      if (!diag) {
        double2 b = rb[q];
        if (has_phase) {
          double2 const p = phase[s & 1][kk];
          b = make_double2(p.x * b.x - p.y * b.y, p.x * b.y + p.y * b.x);
        }
        Bs[kk][row + 16 * q] = b;
      }
    }
    int32_t const h = static_cast<int32_t>(s / spp);
    bool const last = s + 1 == s1 || (s + 1) % spp == 0;  // the plane (or the share) ends here
    if (last && tid < kOps && tid < f.n_ops) {
      double c, sn;
      unit(static_cast<int64_t>(f.k[tid]) * h, f.n_planes, &c, &sn);
      turn[tid] = make_double2(c, sn);
    }
    __syncthreads();
    if (s + 1 < s1) fetch(s + 1);
    if (warp_on) {
      double2 const *a_row = &As[0][kB * bi];
      double2 const *b_row = diag ? &As[0][kB * bj] : &Bs[0][kB * bj];
#pragma unroll 4
      for (int k = 0; k < kK; ++k) {
        double2 a[kB], b[kB];
#pragma unroll
        for (int q = 0; q < kB; ++q) {
          a[q] = a_row[k * kLd + q];
          b[q] = b_row[k * kLd + q];
        }
#pragma unroll
        for (int e = 0; e < kE; ++e) mac(acc[e], a[e % kB], b[e / kB]);
      }
      if (last) {
        // sum += G e^{-i phi}: re = g.x c + g.y s, im = g.y c - g.x s; the
        // Hermitian sums keep the four products apart, which give the sum
        // with e^{+i phi} (the entries below the diagonal) as well.
#pragma unroll
        for (int o = 0; o < kOps; ++o) {
          double const c = o < f.n_ops ? turn[o].x : 0, sn = o < f.n_ops ? turn[o].y : 0;
#pragma unroll
          for (int e = 0; e < kE; ++e) {
            if (kHerm) {
              sum[o][e][0] = fma(acc[e].x, c, sum[o][e][0]);
              sum[o][e][1] = fma(acc[e].y, sn, sum[o][e][1]);
              sum[o][e][kSums - 2] = fma(acc[e].y, c, sum[o][e][kSums - 2]);
              sum[o][e][kSums - 1] = fma(acc[e].x, sn, sum[o][e][kSums - 1]);
            } else {
              sum[o][e][0] = fma(acc[e].x, c, fma(acc[e].y, sn, sum[o][e][0]));
              sum[o][e][1] = fma(acc[e].y, c, fma(-acc[e].x, sn, sum[o][e][1]));
            }
          }
        }
#pragma unroll
        for (int e = 0; e < kE; ++e) acc[e] = make_double2(0, 0);
      }
    }
  }

  // Partial sums of the cluster's CTAs, added in rank order; rank r finishes
  // the blocks r kThr / split .. of the tile.
  cg::cluster_group cluster = cg::this_cluster();
#pragma unroll
  for (int o = 0; o < kOps; ++o) {
    if (o >= f.n_ops) break;
    __syncthreads();  // operands, or the previous operator's sums, are consumed
#pragma unroll
    for (int e = 0; e < kE; ++e)
#pragma unroll
      for (int s = 0; s < kSums; ++s) smem[(e * kSums + s) * kThr + blk] = sum[o][e][s];
    if (split > 1)
      cluster.sync();
    else
      __syncthreads();
    int const n_slot = kThr / split;
    for (int it = tid; it < kE * n_slot; it += kThr) {
      int const slot = rank * n_slot + it % n_slot, e = it / n_slot;
      if (slot >= n_act) continue;
      double r[kSums];
#pragma unroll
      for (int s = 0; s < kSums; ++s) r[s] = 0;
      for (int q = 0; q < split; ++q) {
        double const *src = split > 1 ? cluster.map_shared_rank(smem, q) : smem;
#pragma unroll
        for (int s = 0; s < kSums; ++s) r[s] += src[(e * kSums + s) * kThr + slot];
      }
      int ci = 0, cj = 0;
      if (diag) {
        while ((cj + 1) * (cj + 2) / 2 <= slot) ++cj;
        ci = slot - cj * (cj + 1) / 2;
      } else {
        ci = slot % nbi;
        cj = slot / nbi;
      }
      int const i = i0 + kB * ci + e % kB, j = j0 + kB * cj + e / kB;
      if (i >= nev || j >= nev || (kHerm && i > j)) continue;
      int32_t const op = op_ids ? op_ids[f.op[o]] : f.op[o];
      double2 *out = vdv + (static_cast<int64_t>(2 * op) * g.Lt + t) * nev * nev;
      int64_t const at = i + static_cast<int64_t>(nev) * j, mt = j + static_cast<int64_t>(nev) * i;
      if (kHerm) {
        out[at] = make_double2(r[0] + r[1], r[kSums - 2] - r[kSums - 1]);
        if (i != j) out[mt] = make_double2(r[0] - r[1], -(r[kSums - 2] + r[kSums - 1]));
      } else if (f.dag[o]) {
        out[mt] = make_double2(r[0], -r[1]);
      } else {
        out[at] = make_double2(r[0], r[1]);
      }
    }
    if (split > 1) cluster.sync();  // remote sums are read before they are overwritten
  }
}

int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    sms = 1;
  return sms;
}

int64_t tiles_of(int32_t nev, int32_t side, bool herm) {
  int64_t const n = (nev + side - 1) / side;
  return herm ? n * (n + 1) / 2 : n * n;
}

template <int kB, bool kHerm, int kOps, bool kW>
cudaError_t launch_tiles(double2 *vdv, double2 const *V, double2 const *W, FamilyArgs const &args,
                         int32_t n_fam, int32_t const *op_ids, int32_t t0, int32_t nt,
                         int32_t v_t0, Geometry const &g, cudaStream_t stream) {
  int64_t const tiles = tiles_of(g.nev, 16 * kB, kHerm);
  int64_t const steps = (g.dim_row + kK - 1) / kK;
  // Cluster size: 12 CTAs per SM over the launch (six rounds of two resident
  // ones, so that the last, partly idle round is a small share), at least 16
  // steps per CTA.
  int64_t const ctas = tiles * n_fam * nt, want = 12LL * sm_count();
  int32_t split = 1;
  while (split < 8 && ctas * split < want && steps >= 32LL * split) split *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles * split), static_cast<unsigned>(n_fam),
                     static_cast<unsigned>(nt));
  cfg.blockDim = dim3(kThr);
  cfg.stream = stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = static_cast<unsigned>(split);
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaError_t const e = cudaLaunchKernelEx(&cfg, vdv_family_kernel<kB, kHerm, kOps, kW>, vdv, V,
                                           W, args, op_ids, t0, v_t0, split, g);
  return e != cudaSuccess ? e : cudaGetLastError();
}

// Two by two entries per thread (32 x 32 tiles) read half the shared memory of
// one entry per thread; 16 x 16 tiles are for launches that would not give
// every SM two CTAs even with clusters of 8.
template <bool kHerm, int kOps, bool kW>
cudaError_t launch(double2 *vdv, double2 const *V, double2 const *W, FamilyArgs const &args,
                   int32_t n_fam, int32_t const *op_ids, int32_t t0, int32_t nt, int32_t v_t0,
                   Geometry const &g, cudaStream_t stream) {
  for (int32_t z = 0; z < nt; z += 65535) {
    int32_t const nz = std::min(nt - z, 65535);
    bool const few = 8 * tiles_of(g.nev, 32, kHerm) * n_fam * nz < 2LL * sm_count();
    cudaError_t const e =
        few ? launch_tiles<1, kHerm, kOps, kW>(vdv, V, W, args, n_fam, op_ids, t0 + z, nz, v_t0, g,
                                               stream)
            : launch_tiles<2, kHerm, kOps, kW>(vdv, V, W, args, n_fam, op_ids, t0 + z, nz, v_t0, g,
                                               stream);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace

cudaError_t vdaggerv_fp64(double2 *vdv, double2 const *V, VdvFamily const *fam, int32_t n_fam,
                          int32_t t0, int32_t nt, Geometry g, cudaStream_t stream,
                          int32_t v_t0) {
  if (n_fam == 0 || nt == 0) return cudaSuccess;
  for (int herm = 0; herm < 2; ++herm)
    for (int ops = 1; ops <= kVdvFp64Ops; ++ops) {
      FamilyArgs args{};
      int32_t n = 0;
      for (int32_t k = 0; k <= n_fam; ++k) {
        bool const mine = k < n_fam && (fam[k].herm != 0) == (herm != 0) && fam[k].n_ops == ops;
        if (mine) args.f[n++] = fam[k];
        if (n == kMaxFam || (k == n_fam && n > 0)) {
          cudaError_t e = cudaErrorInvalidValue;
          auto run = [&](auto h, auto o) {
            return launch<decltype(h)::value, decltype(o)::value, false>(
                vdv, V, nullptr, args, n, nullptr, t0, nt, v_t0, g, stream);
          };
          std::integral_constant<bool, true> const H{};
          std::integral_constant<bool, false> const N{};
          std::integral_constant<int, 1> const one{};
          std::integral_constant<int, 2> const two{};
          std::integral_constant<int, 3> const three{};
          if (herm)
            e = ops == 1 ? run(H, one) : ops == 2 ? run(H, two) : run(H, three);
          else
            e = ops == 1 ? run(N, one) : ops == 2 ? run(N, two) : run(N, three);
          if (e != cudaSuccess) return e;
          n = 0;
        }
      }
    }
  return cudaSuccess;
}

cudaError_t vdaggerv_fp64_w(double2 *vdv, double2 const *V, double2 const *W, int32_t const *op,
                            int32_t t, Geometry g, cudaStream_t stream, int32_t v_t0) {
  FamilyArgs args{};
  VdvFamily &f = args.f[0];
  f.axis = 3;
  f.n_planes = 1;
  f.sgn = 1;
  f.n_ops = 1;
  f.op[0] = 0;  // index into op
  return launch<false, 1, true>(vdv, V, W, args, 1, op, t, 1, v_t0, g, stream);
}

}  // namespace dev
}  // namespace slaph
