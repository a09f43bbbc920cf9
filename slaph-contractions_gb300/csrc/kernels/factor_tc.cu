// Diluted factors Q1 and Q2 on the tensor cores (tcgen05, sm_103a).
//
// The factor builders of src/DilutedFactorFactory.cpp are products over the
// eigenvector index with K = nev:
//   Q2M[t,b1,r1,vdv](a, bd nev + v) = sum_w conj(P_r1((4t+bd) nev + w, b1 eds + a)) VdV_t(w, v)
//     (:200-218; one dense GEMM per timeslice: perambulator rows x VdaggerV columns)
//   X1[t](r a, (r2 b d) c) = sum_v Q1R_r(a, v) P_r2((4t+d) nev + v, b eds + c)
//     (:146-164 for all four Dirac blocks d at once; Q1 picks one block per row
//      block and scales it by the gamma phase)
//   Q2(a, c) = sum_bd sum_v s(bd, a) Gval[bd] Q2M_m(a, bd nev + v) P_r2((4t+Grow[bd]) nev + v, b2 eds + c)
//     (:221-243 with K = (bd, v), the gamma_5 signs s folded into the rows and
//      the gamma phases into the columns)
// They run on the split-BF16 tile pipeline of tc_common.cuh (the GEMM kernel
// of trace_tc.cu, whose epilogue writes dense double-float outputs).  Operand
// rows and columns are gathered from up to four strided segments of a source
// array, each with an exact factor +-1, +-i, and cut into slices here; K is
// padded with zeros to whole k-tiles.
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.cuh"
#include "tc_common.cuh"

namespace slaph {
namespace dev {

__constant__ int32_t c_gamma_row_tc[16][4];
__constant__ int32_t c_gamma_phase_tc[16][4];

namespace {

using namespace tc;

constexpr int kGThreads = 256;

__device__ __forceinline__ unsigned long long absbits(double2 v) {
  unsigned long long const a = __double_as_longlong(v.x) & 0x7FFFFFFFFFFFFFFFULL;
  unsigned long long const b = __double_as_longlong(v.y) & 0x7FFFFFFFFFFFFFFFULL;
  return a > b ? a : b;
}
__device__ __forceinline__ unsigned long long absbits(float4 v) {
  unsigned int const a = __float_as_uint(v.x) & 0x7FFFFFFFu;
  unsigned int const b = __float_as_uint(v.z) & 0x7FFFFFFFu;
  return a > b ? a : b;
}
__device__ __forceinline__ int expo_of(unsigned long long b, double2 const *) {
  return expo_of_absbits64(b);
}
__device__ __forceinline__ int expo_of(unsigned long long b, float4 const *) {
  return expo_of_absbits(static_cast<unsigned int>(b));
}
__device__ __forceinline__ void to_fixed(double2 v, int e, long long &fr, long long &fi) {
  fr = fixed55(v.x, e);
  fi = fixed55(v.y, e);
}
__device__ __forceinline__ void to_fixed(float4 v, int e, long long &fr, long long &fi) {
  fr = fixed55f(v.x, e) + fixed55f(v.y, e);
  fi = fixed55f(v.z, e) + fixed55f(v.w, e);
}

// Eight consecutive operand rows (A) or columns (B) per CTA (GVecGroup): the
// exponent of each one's largest |re|, |im| over all segments, then the slices
// of (conj?)(factor x value).  In a k-tile, lane (r, kg) = (lane % 8, lane / 8)
// takes the entries 4 kg .. 4 kg + 3 of row r, so that strided rows (adjacent in
// memory) and unit-stride ones both read whole sectors; the A rows of a
// complex row are a row pair, stored by the lanes that shuffles give its words
// (as in the VdaggerV slicing), so that every slice store of a warp fills 512
// contiguous bytes.  One row per CTA with 4-byte stores took 8.1 ms at 24^3x48
// Nev 120, eight rows 4.6.
//
// kRel: a relative source (Q2M).  The product of a perambulator and VdaggerV may
// leave the range of FP32 where Q2, with the second perambulator, does not; its
// segments keep the exponents of their perambulator rows apart, which the row's
// exponent takes in.
template <bool kIsA, typename T, bool kRel = false>
__global__ void __launch_bounds__(kGThreads)
    gvec_slice_kernel(uint8_t *scratch, int32_t *expo, GVecGroup const *groups, GVec const *items,
                      T const *src, int32_t k_tiles, int32_t conj) {
  constexpr int kWarps = kGThreads / 32, kWords = sizeof(GVec) / 4;
  __shared__ GVec it[8];
  __shared__ unsigned long long red[kWarps][8];
  GVecGroup const gr = groups[blockIdx.x];
  for (int w = threadIdx.x; w < gr.n * kWords; w += kGThreads)
    reinterpret_cast<uint32_t *>(it)[w] =
        reinterpret_cast<uint32_t const *>(items + gr.first)[w];
  __syncthreads();
  // kRel: the exponents of the segments' rows, biased, in the place of their indices.
  // The bits of a value's magnitude plus 2^23 times that order the values of all
  // segments and hold the (biased) exponent from bit 23 on.
  constexpr int kRelBias = 4096;
  if (kRel) {
    static_assert(8 * kGMaxSeg <= kGThreads, "one thread per segment");
    int const i = threadIdx.x / kGMaxSeg, s = threadIdx.x % kGMaxSeg;
    if (i < gr.n && s < it[i].n_seg)
      it[i].seg[s].e_row = expo[it[i].seg[s].e_row] + kRelBias;
    __syncthreads();
  }
  int const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  int const r = lane % 8, kg = lane / 8;
  bool const on = r < gr.n;
  GVec const &v = it[on ? r : 0];
  int const len = v.seg_len, K = v.n_seg * len;
  auto load = [&](int k, int &s) {
    s = (k >= len) + (k >= 2 * len) + (k >= 3 * len);
    return src[v.seg[s].src + static_cast<int64_t>(k - s * len) * v.stride];
  };
  unsigned long long mx = 0;
  for (int kt = warp; kt < k_tiles; kt += kWarps)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int const k = kt * (kTK / 2) + 4 * kg + q;
      int s;
      if (on && k < K) {
        unsigned long long b = absbits(load(k, s));
        if (kRel && b != 0)
          b += static_cast<unsigned long long>(v.seg[s].e_row) << 23;
        mx = b > mx ? b : mx;
      }
    }
#pragma unroll
  for (int o = 8; o <= 16; o <<= 1) {
    unsigned long long const y = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = y > mx ? y : mx;
  }
  if (kg == 0) red[warp][r] = mx;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kWarps; ++w) mx = red[w][r] > mx ? red[w][r] : mx;
  int const e = !kRel    ? expo_of(mx, src)
                : mx != 0 ? static_cast<int>(mx >> 23) - 126 - kRelBias
                          : 0;
  if (warp == 0 && kg == 0 && on) expo[v.expo] = e;
  uint8_t *region = scratch + it[0].dst;
  int const row0 = it[0].row;  // a multiple of 8
  for (int kt = warp; kt < k_tiles; kt += kWarps) {
    uint32_t w[kSlices][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int const k = kt * (kTK / 2) + 4 * kg + q;
      long long fr = 0, fi = 0;
      if (on && k < K) {
        int s;
        T const x = load(k, s);
        to_fixed(x, kRel ? e + kRelBias - v.seg[s].e_row : e, fr, fi);
        long long const re = fr, im = fi;
        switch (v.seg[s].factor & 3) {
          case 1: fr = -im; fi = re; break;   // x i
          case 2: fr = -re; fi = -im; break;  // x -1
          case 3: fr = im; fi = -re; break;   // x -i
          default: break;
        }
        if (conj) fi = -fi;
      }
      float dre[kSlices], dim[kSlices];
      digits6(fr, dre);
      digits6(fi, dim);
#pragma unroll
      for (int p = 0; p < kSlices; ++p) w[p][q] = bf16x2(dre[p], dim[p]);
    }
    if (kIsA) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // the two core-matrix groups of the 16 A rows
        int const ir = 4 * h + r / 2;  // the complex row that this lane stores
        int const i = row0 + ir;
        int const arow = 2 * (i % (kTM / 2)) + (r & 1);
        uint8_t *dst = region +
                       (static_cast<int64_t>(i / (kTM / 2)) * k_tiles + kt) * kStageA +
                       ((arow >> 3) * 4 + kg) * 128 + (arow & 7) * 16;
#pragma unroll
        for (int p = 0; p < kSlices; ++p) {
          uint32_t x[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t const y = __shfl_sync(0xffffffffu, w[p][q], ir + 8 * kg);
            x[q] = (r & 1) ? __byte_perm(y, 0, 0x1032) ^ 0x8000u : y;
          }
          if (ir < gr.n)
            *reinterpret_cast<uint4 *>(dst + p * kABlk) = make_uint4(x[0], x[1], x[2], x[3]);
        }
      }
    } else if (on) {
      int const c = row0 + r, rr = c % kTN;
      uint8_t *dst = region + (static_cast<int64_t>(c / kTN) * k_tiles + kt) * kStageB +
                     ((rr >> 3) * 4 + kg) * 128 + (rr & 7) * 16;
#pragma unroll
      for (int p = 0; p < kSlices; ++p)
        *reinterpret_cast<uint4 *>(dst + p * kBBlk) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
    }
  }
}

__device__ __forceinline__ float4 phase_mul(int code, float4 v) {
  switch (code & 3) {
    case 1: return make_float4(-v.z, -v.w, v.x, v.y);
    case 2: return make_float4(-v.x, -v.y, -v.z, -v.w);
    case 3: return make_float4(v.z, v.w, -v.x, -v.y);
    default: return v;
  }
}

// Entry (a, c) of a factor: Q1 (src/DilutedFactorFactory.cpp:146-164) from X1 is
// gamma_phase[row] X1[row0 + a, col0 + Grow[row] eds + c] with row = a / dilE; Q2
// from its GEMM output y[off + a + ld c].
__device__ __forceinline__ float4 entry(Q1Gather const &q, float4 const *x, int a, int c, int eds) {
  int const row = a / (eds / 4);
  float4 const v = x[q.x_off + (q.row0 + a) +
                     static_cast<int64_t>(q.ld) *
                         (q.col0 + c_gamma_row_tc[q.gamma][row] * eds + c)];
  return phase_mul(c_gamma_phase_tc[q.gamma][row], v);
}
__device__ __forceinline__ float4 entry(Q2Gather const &q, float4 const *y, int a, int c, int) {
  return y[q.off + a + static_cast<int64_t>(q.ld) * c];
}

// One CTA per factor slot, in chunks of up to 32 rows: entries are read along
// a, where the source is contiguous, and pass through shared memory for the
// transposed layout, so that the stores of both layouts fill whole lines.
// Memory-bound: 16 bytes read and 16 written per entry and layout (with the
// transposed stores straight from registers, 32 lanes a line each, 24^3x48
// Nev 120 took 7.1 ms against 2.1).
constexpr int kGatherRows = 32;
template <typename G>
__global__ void __launch_bounds__(256)
    gather_kernel(float4 *sn, float4 *st, unsigned int *slot_bits, G const *g, float4 const *src,
                  int32_t eds) {
  __shared__ float4 tile[64 * (kGatherRows + 1)];
  __shared__ unsigned int red[8];
  G const q = g[blockIdx.x];
  int64_t const at = static_cast<int64_t>(q.slot) * eds * eds;
  unsigned int mx = 0;
  for (int a0 = 0; a0 < eds; a0 += kGatherRows) {
    int const ra = min(kGatherRows, eds - a0), n = ra * eds;
    for (int k = threadIdx.x; k < n; k += 256) {
      int const a = k % ra, c = k / ra;
      float4 const v = entry(q, src, a0 + a, c, eds);
      mx = max(mx, max(__float_as_uint(v.x) & 0x7FFFFFFFu, __float_as_uint(v.z) & 0x7FFFFFFFu));
      if (q.need & 1) sn[at + a0 + a + eds * c] = v;
      if (q.need & 2) tile[c * (kGatherRows + 1) + a] = v;
    }
    if (q.need & 2) {
      __syncthreads();
      for (int k = threadIdx.x; k < n; k += 256) {
        int const c = k % eds, a = k / eds;
        st[at + c + eds * (a0 + a)] = tile[c * (kGatherRows + 1) + a];
      }
      __syncthreads();
    }
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) mx = max(mx, red[w]);
    slot_bits[q.slot] = mx;
  }
}

}  // namespace

cudaError_t upload_gamma_tc(cudaStream_t stream) {
  int32_t row[16][4], ph[16][4];
  for (int m = 0; m < 16; ++m)
    for (int c = 0; c < 4; ++c) {
      row[m][c] = gamma_row_host(m, c);
      ph[m][c] = gamma_phase_host(m, c);
    }
  cudaError_t e = cudaMemcpyToSymbolAsync(c_gamma_row_tc, row, sizeof row, 0,
                                          cudaMemcpyHostToDevice, stream);
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbolAsync(c_gamma_phase_tc, ph, sizeof ph, 0, cudaMemcpyHostToDevice,
                                 stream);
}

cudaError_t gvec_slice_f64(uint8_t *scratch, int32_t *expo, GVecGroup const *groups, int64_t n,
                           GVec const *items,
                           bool is_a, bool conj, double2 const *src, int32_t k_tiles,
                           cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  if (is_a)
    gvec_slice_kernel<true, double2><<<static_cast<unsigned>(n), kGThreads, 0, stream>>>(
        scratch, expo, groups, items, src, k_tiles, conj ? 1 : 0);
  else
    gvec_slice_kernel<false, double2><<<static_cast<unsigned>(n), kGThreads, 0, stream>>>(
        scratch, expo, groups, items, src, k_tiles, conj ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t gvec_slice_df(uint8_t *scratch, int32_t *expo, GVecGroup const *groups, int64_t n,
                           GVec const *items,
                          bool is_a, bool conj, float4 const *src, int32_t k_tiles,
                          cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  if (is_a)
    gvec_slice_kernel<true, float4><<<static_cast<unsigned>(n), kGThreads, 0, stream>>>(
        scratch, expo, groups, items, src, k_tiles, conj ? 1 : 0);
  else
    gvec_slice_kernel<false, float4><<<static_cast<unsigned>(n), kGThreads, 0, stream>>>(
        scratch, expo, groups, items, src, k_tiles, conj ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t gvec_slice_relative(uint8_t *scratch, int32_t *expo, GVecGroup const *groups,
                                int64_t n, GVec const *items, float4 const *src, int32_t k_tiles,
                                cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  gvec_slice_kernel<true, float4, true><<<static_cast<unsigned>(n), kGThreads, 0, stream>>>(
      scratch, expo, groups, items, src, k_tiles, 1);
  return cudaGetLastError();
}

cudaError_t q1_gather(float4 *sn, float4 *st, unsigned int *slot_bits, Q1Gather const *g,
                      int64_t n, float4 const *x, int32_t dilE, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  if (n > 0x7fffffffLL || dilE > 16) return cudaErrorInvalidValue;
  gather_kernel<<<static_cast<unsigned>(n), 256, 0, stream>>>(sn, st, slot_bits, g, x, 4 * dilE);
  return cudaGetLastError();
}

cudaError_t q2_gather(float4 *sn, float4 *st, unsigned int *slot_bits, Q2Gather const *g,
                      int64_t n, float4 const *y, int32_t eds, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  if (n > 0x7fffffffLL || eds > 64) return cudaErrorInvalidValue;
  gather_kernel<<<static_cast<unsigned>(n), 256, 0, stream>>>(sn, st, slot_bits, g, y, eds);
  return cudaGetLastError();
}

int32_t gemm_k_tiles(int64_t K) { return static_cast<int32_t>((K + kTK / 2 - 1) / (kTK / 2)); }

}  // namespace dev
}  // namespace slaph
