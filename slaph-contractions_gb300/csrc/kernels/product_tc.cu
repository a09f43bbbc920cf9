// Diluted-factor products on the tensor cores (tcgen05, sm_103a).
//
// operator* (src/DilutedFactor.cpp:6-51) and multiply<1,1>
// (include/DilutedFactor.hpp:164-187) form C = L R for every compatible pair of
// left and right factor matrices (eds x eds, eds = 4 dilE).  Within one
// dependency level each left matrix meets dozens of right matrices, every one
// with its own set, so the products of a level are grouped by left matrix:
// a group holds 64 / eds left matrices (one 64-row M tile of stacked rows) and
// the union U of their right matrices (eds columns each), and one GEMM
//   D(group row (l, i), column (u, j)) = sum_k L_l(i, k) R_u(k, j)
// gives every product of the group; the epilogue keeps the entries of the
// pairs the level asks for and writes them as double-float matrices into the
// product slots, in the natural or the transposed layout or both, together with the
// largest entry of every slot (for the slicing of the trace operands).
//
// Operands, in the split-BF16 scheme of tc_common.cuh: A rows are the rows of
// the left matrices (conjugated, so that the conjugating form gives the plain
// product), one exponent per row; each distinct right matrix of the level is
// sliced once into a stream of its own, [k-tile][slice][8-column group][512
// bytes] with one exponent per column.
//
// product_step_kernel (eds <= 32) takes one right matrix per step against the
// group's A operand, which stays in shared memory.  Sizes below 16 or 32 are padded
// with zeros in the operands (18^3x48, eds = 24: products 3.8 ms in the double-float
// kernel, 1.5 ms here).  A step is one or two k-tiles, so promotion and epilogue,
// not the MMAs, bound it.  With the
// general tile (tc_common.cuh: 80 columns, eight promotion warps that hold 40
// columns of running sums and hand them to an unrolled epilogue) a tile's MMAs
// took 2.7 us of 14: the code did not fit the instruction cache and nothing
// overlapped.  Here sixteen promotion warps take eight columns each in one
// straight pass (there is one chunk, so no running sums), two accumulator sets
// let the next step's MMAs run meanwhile, a right matrix is one bulk copy, and
// pairs that the level does not ask for are skipped.  24^3x48 Nev 120: 9.8 ->
// 3.8 ms.  Then the stores bound it: a product is written in the layouts in which
// it is read only, its transposed rows in whole sectors: 3.3 ms (one block pair of
// 64 timeslices 3.8 -> 2.8).  eds = 64 does not fit (A alone is 192 KB) and keeps the general
// tile, whose producer gathers the B stage with one copy per (slice, matrix).
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.cuh"
#include "tc_common.cuh"

namespace slaph {
namespace dev {

namespace {

using namespace tc;

constexpr int kPSliceThreads = 256;

// Row group (A: four complex rows = eight A' rows; B: eight columns) of one
// k-tile: lane (r, kc) = (lane / 4, lane % 4) stores the four complex entries
// 4 kc .. 4 kc + 3 of its row as one 16-byte row segment per slice.  v: the
// entries (A: the two that this lane of a row pair cuts, a_row_words), e: the
// row's exponent; A rows are conjugated.
template <bool kIsA>
__device__ __forceinline__ void slice_row_segment(float4 const (&v)[kIsA ? 2 : 4], int e, int r,
                                                  uint8_t *dst, uint32_t blk) {
  uint32_t w[kSlices][4];
  if constexpr (kIsA) {
    a_row_words(v, e, r & 1, w);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float dre[kSlices], dim[kSlices];
      digits6(fixed55f(v[q].x, e) + fixed55f(v[q].y, e), dre);
      digits6(fixed55f(v[q].z, e) + fixed55f(v[q].w, e), dim);
#pragma unroll
      for (int s = 0; s < kSlices; ++s) w[s][q] = bf16x2(dre[s], dim[s]);
    }
  }
#pragma unroll
  for (int s = 0; s < kSlices; ++s)
    *reinterpret_cast<uint4 *>(dst + s * blk) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
}

// Largest |re|, |im| (high words) of the lanes' entries, over the lanes whose
// bits `mask` differ (the lanes of one row).
template <int N>
__device__ __forceinline__ unsigned int row_max(float4 const (&v)[N], unsigned int mx,
                                                int mask) {
#pragma unroll
  for (int q = 0; q < N; ++q)
    mx = max(mx, max(__float_as_uint(v[q].x) & 0x7FFFFFFFu, __float_as_uint(v[q].z) & 0x7FFFFFFFu));
#pragma unroll
  for (int o = 1; o <= 4; o <<= 1)
    if (mask & o) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  return mx;
}

// A regions: one CTA per group; the group's 64 rows (left matrix l = row /
// eds, row i = row % eds, read from the transposed layout where rows are
// contiguous) in quads of four rows, warp w taking quads w, w + 8.  Rows of
// absent left matrices are not written (the epilogue skips them).
__global__ void __launch_bounds__(kPSliceThreads)
    prod_slice_a_kernel(uint8_t *scratch, int32_t *expo, ProdGroup const *groups,
                        float4 const *slots_t, int32_t eds, int64_t a_bytes) {
  ProdGroup const gr = groups[blockIdx.x];
  int64_t const ms = static_cast<int64_t>(eds) * eds;
  int const pad = prod_tc_pad(eds), k_tiles = pad / (kTK / 2);
  int const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  int const r = lane / 4, kc = lane % 4;
  uint8_t *region = scratch + static_cast<int64_t>(blockIdx.x) * a_bytes;
  for (int quad = warp; quad < (kTM / 2) / 4; quad += kPSliceThreads / 32) {
    int const cr = 4 * quad + r / 2;  // complex row of the M tile
    int const l = cr / pad, i = cr % pad;
    if (l >= gr.n_l) continue;  // warp-uniform: a quad lies inside one matrix
    float4 const *src =
        slots_t + static_cast<int64_t>(groups[blockIdx.x].l[l]) * ms + static_cast<int64_t>(i) * eds;
    // the two entries of a k-tile that this lane cuts (zero in the padding)
    auto load = [&](int kt, float4 (&v)[2]) {
      int const k0 = kt * (kTK / 2) + 4 * kc + 2 * (r & 1);
#pragma unroll
      for (int q = 0; q < 2; ++q)
        v[q] = i < eds && k0 < eds ? src[k0 + q] : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    unsigned int mx = 0;
    for (int kt = 0; kt < k_tiles; ++kt) {
      float4 v[2];
      load(kt, v);
      mx = row_max(v, mx, 1 | 2 | 4);
    }
    // |hi + lo| < 2^e whenever |hi| < 2^e (|lo| <= ulp(hi) / 2).
    int const e = wide_expo(mx);  // K' = 2 eds <= 128
    if (lane % 8 == 0) expo[gr.ea + cr] = e;
    int const arow = 2 * cr + (r & 1);
    uint8_t *base = region + ((arow >> 3) * 4 + kc) * 128 + (arow & 7) * 16;
    for (int kt = 0; kt < k_tiles; ++kt) {
      float4 v[2];
      load(kt, v);
      slice_row_segment<true>(v, e, r, base + static_cast<int64_t>(kt) * kStageA, kABlk);
    }
  }
}

// Right-matrix streams: one CTA per distinct right matrix of the level, warp w
// taking the 8-column groups w, w + 8, ... (columns read from the natural
// layout, where they are contiguous).
__global__ void __launch_bounds__(kPSliceThreads)
    prod_slice_r_kernel(uint8_t *streams, int32_t *expo, int32_t const *r_slots,
                        float4 const *slots_n, int32_t eds) {
  int64_t const ms = static_cast<int64_t>(eds) * eds;
  int const pad = prod_tc_pad(eds), k_tiles = pad / (kTK / 2), n_cg = pad / 8;
  int const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  int const r = lane / 4, kc = lane % 4;
  uint8_t *stream = streams + static_cast<int64_t>(blockIdx.x) * prod_tc_r_bytes(eds);
  float4 const *mat = slots_n + static_cast<int64_t>(r_slots[blockIdx.x]) * ms;
  for (int cg = warp; cg < n_cg; cg += kPSliceThreads / 32) {
    int const j = 8 * cg + r;
    float4 const *src = mat + static_cast<int64_t>(j) * eds;
    auto load = [&](int kt, float4 (&v)[4]) {
      int const k0 = kt * (kTK / 2) + 4 * kc;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        v[q] = j < eds && k0 < eds ? src[k0 + q] : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    unsigned int mx = 0;
    for (int kt = 0; kt < k_tiles; ++kt) {
      float4 v[4];
      load(kt, v);
      mx = row_max(v, mx, 1 | 2);
    }
    int const e = wide_expo(mx);  // K' = 2 eds <= 128
    if (kc == 0) expo[static_cast<int64_t>(blockIdx.x) * pad + j] = e;
    for (int kt = 0; kt < k_tiles; ++kt) {
      float4 v[4];
      load(kt, v);
      // [k-tile][slice][8-column group][512 B]: a slice step is n_cg groups
      uint8_t *dst = stream + ((static_cast<int64_t>(kt) * kSlices * n_cg + cg) * 4 + kc) * 128 +
                     r * 16;
      slice_row_segment<false>(v, e, r, dst, static_cast<uint32_t>(n_cg) * 512u);
    }
  }
}

// Stage loader of the product GEMM: the group's A block (lane 0) and the B
// stage gathered from the right-matrix streams, one copy per (slice, right
// matrix) spread over the lanes; padding columns of a group's last tile are not
// copied (the epilogue skips them).
struct ProdTiles {
  uint8_t const *scratch;  // A regions from 0, right-matrix streams from r_off
  int64_t a_bytes, r_off;
  ProdTile const *tiles;
  ProdGroup const *groups;
  int32_t const *u_list;  // right-matrix index of each group column block
  int32_t eds, k_tiles;
  // One tile's copies: the A block, and per lane up to two B copies (one per
  // (slice, right matrix overlapping the tile): its columns are contiguous
  // both in its stream and in the stage), addresses of k-tile 0.
  struct Ctx {
    uint8_t const *a;
    uint8_t const *src[2];
    uint32_t dst[2], bytes[2];
    uint32_t tx;
  };
  __device__ __forceinline__ Ctx context(int i, int lane) const {
    ProdTile const t = tiles[i];
    ProdGroup const gr = groups[t.group];
    Ctx c;
    c.a = scratch + t.group * a_bytes;
    int const c0 = t.nt * kTN;
    int const cols = min(kTN, eds * gr.n_u - c0);  // a multiple of 8
    c.tx = kStageA + static_cast<uint32_t>(kSlices * cols) * 64u;
    int64_t const r_bytes = prod_tc_r_bytes(eds);
    int const r_cg = eds / 8, u0 = c0 / eds, n_blk = (c0 + cols - 1) / eds - u0 + 1;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int const q = lane + 32 * h;
      c.bytes[h] = 0;
      c.src[h] = scratch;
      c.dst[h] = 0;
      if (q < kSlices * n_blk) {
        int const s = q / n_blk, u = u0 + q % n_blk;
        int const cs = max(c0, u * eds), ce = min(c0 + cols, (u + 1) * eds);
        c.src[h] = scratch + r_off + u_list[gr.u_off + u] * r_bytes +
                   (static_cast<int64_t>(s) * r_cg + (cs - u * eds) / 8) * 512;
        c.dst[h] = kStageA + s * kBBlk + ((cs - c0) / 8) * 512;
        c.bytes[h] = static_cast<uint32_t>(ce - cs) * 64u;
      }
    }
    return c;
  }
  __device__ __forceinline__ void load(Ctx const &c, int kt, uint8_t *dst, uint64_t *bar,
                                       int lane) const {
    if (lane == 0) {
      mbar_expect_tx(bar, c.tx);
      bulk_g2s(dst, c.a + static_cast<int64_t>(kt) * kStageA, kStageA, bar);
    }
    __syncwarp();
    // k-tile step of a stream: kSlices x eds columns x 64 bytes
    int64_t const kt_off = static_cast<int64_t>(kt) * kSlices * eds * 64;
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (c.bytes[h]) bulk_g2s(dst + c.dst[h], c.src[h] + kt_off, c.bytes[h], bar);
  }
};

// Epilogue: A' row 2 cr + (re | im), cr = l eds + i; column c = u eds + j.
// A warp's 32 rows lie in one left matrix l.  Before the tile is promoted,
// lane k fetches the product slot and the column exponent of the warp's
// columns k and 32 + k; the column loop takes them by warp shuffles.
// The even lane of each row pair holds Re, the odd one Im; after one exchange
// the even lane writes the natural layout and the odd lane the transposed one.
struct ProdEpilogue {
  ProdTiles tl;
  int32_t const *expo;    // A rows from 0 (64 per group), right columns from r_expo
  int64_t r_expo;
  int32_t const *out_tab;  // [group column block][4]: product slot per left matrix
  float4 *slots_n, *slots_t;
  unsigned int *slot_bits;  // largest |re|, |im| per slot (float bits), by atomicMax
  struct Pre {
    int ok, er, cbase;
    int slot0, ec0, slot1, ec1;
  };
  __device__ __forceinline__ Pre prepare(int it, int row, int col0) const {
    Pre p{0, 0, 0, -1, 0, -1, 0};
    ProdTile const t = tl.tiles[it];
    ProdGroup const gr = tl.groups[t.group];
    int const eds = tl.eds, lane = threadIdx.x % 32;
    int const cr = row / 2, l = cr / eds;
    p.cbase = t.nt * kTN + col0;
    if (l >= gr.n_l) return p;  // warp-uniform
    p.ok = 1;
    p.er = expo[gr.ea + cr];
    int const ncols = eds * gr.n_u;
    auto meta = [&](int c, int &slot, int &ec) {
      if (c >= ncols) return;
      int const u = c / eds;
      slot = out_tab[4 * (gr.u_off + u) + l] >> 2;  // both layouts are written
      ec = expo[r_expo + static_cast<int64_t>(tl.u_list[gr.u_off + u]) * eds + c % eds];
    };
    meta(p.cbase + lane, p.slot0, p.ec0);
    if (lane < kColsW - 32) meta(p.cbase + 32 + lane, p.slot1, p.ec1);
    return p;
  }
  __device__ __forceinline__ void operator()(Pre const &p, int, int row, int,
                                             float const (&hi)[kColsW],
                                             float const (&lo)[kColsW]) const {
    if (!p.ok) return;  // warp-uniform
    int const eds = tl.eds;
    int64_t const ms = static_cast<int64_t>(eds) * eds;
    int const i = (row / 2) % eds;
    // The slot of a column is the same for the whole warp (one left matrix):
    // the largest |hi| of a run of columns of one slot goes to slot_bits by
    // one warp reduction and one atomic.
    int run_slot = -1;
    unsigned int run_max = 0;
    auto flush = [&] {
      unsigned int const m = __reduce_max_sync(0xffffffffu, run_max);
      if (run_slot >= 0 && (threadIdx.x % 32) == 0) atomicMax(slot_bits + run_slot, m);
    };
#pragma unroll
    for (int cc = 0; cc < kColsW; ++cc) {
      int const slot = __shfl_sync(0xffffffffu, cc < 32 ? p.slot0 : p.slot1, cc % 32);
      int const ec = __shfl_sync(0xffffffffu, cc < 32 ? p.ec0 : p.ec1, cc % 32);
      int const sh = max(p.er + ec - 14, -252);
      float const h = scale2(hi[cc], sh), lw = scale2(lo[cc], sh);
      float const oh = __shfl_xor_sync(0xffffffffu, h, 1);
      float const ol = __shfl_xor_sync(0xffffffffu, lw, 1);
      if (slot != run_slot) {  // warp-uniform
        flush();
        run_slot = slot;
        run_max = 0;
      }
      if (slot < 0) continue;
      run_max = max(run_max, __float_as_uint(h) & 0x7FFFFFFFu);
      int const j = (p.cbase + cc) % eds;
      if ((row & 1) == 0)
        slots_n[slot * ms + i + static_cast<int64_t>(eds) * j] = make_float4(h, lw, oh, ol);
      else
        slots_t[slot * ms + j + static_cast<int64_t>(eds) * i] = make_float4(oh, ol, h, lw);
    }
    flush();
  }
};

__global__ void __launch_bounds__(kThreads, 1)
    product_gemm_kernel(ProdTiles tl, int32_t n_tiles, int32_t const *expo, int64_t r_expo,
                        int32_t const *out_tab, float4 *slots_n, float4 *slots_t,
                        unsigned int *slot_bits, int *err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  ProdEpilogue epi{tl, expo, r_expo, out_tab, slots_n, slots_t, slot_bits};
  ozaki_tiles(smem, n_tiles, tl.k_tiles, tl, err, epi);
}

// ---------------------------------------------------------------- steps
constexpr int kStepWarps = 16;  // promotion warps: quadrant w % 4, column block w / 4
constexpr int kStepThreads = 32 * (kStepWarps + 2);
constexpr int kStepStages = 4;  // right matrices in flight
constexpr uint32_t kStepTmem = 256;  // columns per accumulator set (6 kPad used)

__host__ __device__ inline uint32_t step_a_bytes(int pad) { return pad / 16 * kStageA; }
__host__ __device__ inline uint32_t step_smem(int pad) {
  return step_a_bytes(pad) + kStepStages * 24u * pad * pad;
}

// Two float4 at a 32-byte boundary in one store (a full sector).
__device__ __forceinline__ void store_pair(float4 *p, float4 const (&v)[2]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0].x),
               "f"(v[0].y), "f"(v[0].z), "f"(v[0].w), "f"(v[1].x), "f"(v[1].y), "f"(v[1].z),
               "f"(v[1].w)
               : "memory");
}

struct StepArgs {
  uint8_t const *scratch;  // A regions from 0, right-matrix streams from r_off
  int64_t a_bytes, r_off;
  ProdTile const *units;
  int32_t n_units;
  int32_t const *u_list;
  int32_t const *expo;  // A rows from 0 (64 per group), right columns from r_expo
  int64_t r_expo;
  int32_t const *out_tab;
  float4 *slots_n, *slots_t;
  unsigned int *slot_bits;
  int *err;
  int32_t eds;
};

template <int kPad>
__global__ void __launch_bounds__(kStepThreads, 1) product_step_kernel(StepArgs const g) {
  constexpr int kKT = kPad / 16;                      // k-tiles
  constexpr uint32_t kRB = 24u * kPad * kPad;         // bytes of a right matrix
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t a_full, a_empty, b_full[kStepStages], b_empty[kStepStages];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], done_bar;
  __shared__ uint32_t tmem_slot;
  int const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  uint8_t *const b_smem = smem + step_a_bytes(kPad);
  if (threadIdx.x == 0) {
    mbar_init(&a_full, 1);
    mbar_init(&a_empty, 1);
    for (int s = 0; s < kStepStages; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], kStepWarps);
    }
    mbar_init(&done_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t const tmem = tmem_slot;

  if (warp == kStepWarps) {  // producer
    bool ok = true;
    uint32_t n_a = 0, n_b = 0;  // A operands, right matrices issued
    for (int i = blockIdx.x; i < g.n_units && ok; i += gridDim.x) {
      ProdTile const t = g.units[i];
      int const idx = lane < t.n ? g.u_list[t.u + lane] : 0;
      if (lane == 0) {
        if (n_a > 0) ok = mbar_wait(&a_empty, (n_a - 1) & 1, g.err, 1);
        if (ok) {
          mbar_expect_tx(&a_full, step_a_bytes(kPad));
          bulk_g2s(smem, g.scratch + t.group * g.a_bytes, step_a_bytes(kPad), &a_full);
        }
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      ++n_a;
      for (int s = 0; s < t.n && ok; ++s) {
        int const r = __shfl_sync(0xffffffffu, idx, s);
        uint32_t const st = n_b % kStepStages, use = n_b / kStepStages;
        if (lane == 0) {
          if (use > 0) ok = mbar_wait(&b_empty[st], (use - 1) & 1, g.err, 1);
          if (ok) {
            mbar_expect_tx(&b_full[st], kRB);
            bulk_g2s(b_smem + st * kRB, g.scratch + g.r_off + static_cast<int64_t>(r) * kRB, kRB,
                     &b_full[st]);
          }
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (ok) ++n_b;
      }
    }
    // All copies have landed before shared memory is released (immediate when
    // the MMA warp consumed them).
    if (lane == 0) {
      if (n_a > 0) mbar_wait(&a_full, (n_a - 1) & 1, g.err, 6);
      for (uint32_t q = n_b > kStepStages ? n_b - kStepStages : 0; q < n_b; ++q)
        mbar_wait(&b_full[q % kStepStages], (q / kStepStages) & 1, g.err, 6);
    }
  } else if (warp == kStepWarps + 1) {
    if (lane == 0) {  // MMA issuer
      bool ok = true;
      uint32_t n_a = 0, n_s = 0;
      uint32_t const a_base = smem_u32(smem);
      for (int i = blockIdx.x; i < g.n_units && ok; i += gridDim.x, ++n_a) {
        int const n = g.units[i].n;
        ok = mbar_wait(&a_full, n_a & 1, g.err, 3);
        for (int s = 0; s < n && ok; ++s, ++n_s) {
          uint32_t const st = n_s % kStepStages, set = n_s % 2;
          ok = mbar_wait(&b_full[st], (n_s / kStepStages) & 1, g.err, 3) &&
               (n_s < 2 || mbar_wait(&acc_empty[set], (n_s / 2 - 1) & 1, g.err, 2));
          if (!ok) break;
          tc_fence_after();
          uint32_t const b_base = smem_u32(b_smem + st * kRB);
          uint32_t const d = tmem + set * kStepTmem;
          // the 21 slice pairs as 9 MMAs per k-step (tc_common.cuh)
#pragma unroll
          for (int ks = 0; ks < 2 * kKT; ++ks) {
#pragma unroll
            for (int p = 0; p < kSlices; ++p) {
#pragma unroll
              for (int q0 = 0; q0 < kSlices - p; q0 += kLevelGroup) {
                int const nb = min(kLevelGroup, kSlices - p - q0);
                uint64_t const ad =
                    smem_desc(a_base + (ks / 2) * kStageA + p * kABlk + (ks % 2) * 256, 128, 512);
                uint64_t const bd = smem_desc(
                    b_base + (ks / 2) * (kSlices * kPad * 64) + q0 * (kPad * 64) + (ks % 2) * 256,
                    128, 512);
                mma_bf16(d + static_cast<uint32_t>((p + q0) * kPad), ad, bd,
                         ks == 0 && p == 0 ? 0u : 1u, idesc_n(nb * kPad));
              }
            }
          }
          mma_commit(&b_empty[st]);
          mma_commit(&acc_full[set]);
        }
        if (ok) mma_commit(&a_empty);
      }
      mma_commit(&done_bar);
      mbar_wait(&done_bar, 0, g.err, 4);
    }
  } else {
    // Promotion: A' row 2 cr + (re | im), cr = l kPad + i; columns 8 blk .. of the
    // step's right matrix.  A warp's rows lie in one left matrix, its columns in
    // one right matrix: one product slot per warp and step.
    int const quad = warp % 4, blk = warp / 4;
    int const row = 32 * quad + lane, cr = row / 2, l = cr / kPad, ri = cr % kPad;
    int const eds = g.eds;
    bool const blk_on = 8 * blk < eds, row_on = ri < eds;
    uint32_t const lane_addr =
        tmem + (static_cast<uint32_t>(32 * quad) << 16) + static_cast<uint32_t>(8 * blk);
    int64_t const ms = static_cast<int64_t>(eds) * eds;
    uint32_t n_s = 0;
    bool ok = true;
    for (int i = blockIdx.x; i < g.n_units && ok; i += gridDim.x) {
      ProdTile const t = g.units[i];
      bool const on = blk_on && l < t.n_l;  // warp-uniform
      // lane s holds the right matrix and the product slot of step s
      int const idx = lane < t.n ? g.u_list[t.u + lane] : 0;
      int const slots = on && lane < t.n ? g.out_tab[4 * (t.u + lane) + l] : -1;
      int const er = on ? g.expo[t.ea + cr] : 0;
      auto column_expo = [&](int s) {  // lane c: exponent of column 8 blk + c of step s
        int const r = __shfl_sync(0xffffffffu, idx, s);
        return blk_on && lane < 8
                   ? g.expo[g.r_expo + static_cast<int64_t>(r) * kPad + 8 * blk + lane]
                   : 0;
      };
      int ec_next = column_expo(0);
      for (int s = 0; s < t.n; ++s, ++n_s) {
        uint32_t const set = n_s % 2;
        int const entry = __shfl_sync(0xffffffffu, slots, s), slot = entry >> 2;
        int const ec_lane = ec_next;
        if (s + 1 < t.n) ec_next = column_expo(s + 1);
        if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[set], (n_s / 2) & 1, g.err, 5))) {
          ok = false;
          break;
        }
        tc_fence_after();
        uint32_t r0[3][8], r1[3][8];
        if (slot >= 0) {  // warp-uniform
          uint32_t const ca = lane_addr + set * kStepTmem;
#pragma unroll
          for (int v = 0; v < 3; ++v) tmem_ld8_issue(ca + static_cast<uint32_t>(v * kPad), r0[v]);
#pragma unroll
          for (int v = 0; v < 3; ++v)
            tmem_ld8_issue(ca + static_cast<uint32_t>((3 + v) * kPad), r1[v]);
          tmem_ld_wait(r0);
          tmem_ld_wait(r1);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[set]);
        if (slot < 0) continue;
        unsigned int mx = 0;
        float4 *const dst = (row & 1) ? g.slots_t + slot * ms + static_cast<int64_t>(eds) * ri
                                      : g.slots_n + slot * ms + ri;
        bool const store = row_on && (entry & ((row & 1) ? 2 : 1)) != 0;
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
          float4 out[2];
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            // the chunk's value in (hi, lo), as in tc_common.cuh
            float s1, x1, s2, x2, s3, x3;
            scaled_sum(__uint_as_float(r0[0][u + y]), __uint_as_float(r0[1][u + y]), 0x1p-8f, s1,
                       x1);
            scaled_sum(s1, __uint_as_float(r0[2][u + y]), 0x1p-16f, s2, x2);
            float const low = fmaf(__uint_as_float(r1[2][u + y]), 0x1p-16f,
                                   fmaf(__uint_as_float(r1[1][u + y]), 0x1p-8f,
                                        __uint_as_float(r1[0][u + y])));
            scaled_sum(s2, low, 0x1p-24f, s3, x3);
            float const e = (x1 + x2) + x3;
            float const hi = s3 + e, lo = e - (hi - s3);
            int const sh = max(er + __shfl_sync(0xffffffffu, ec_lane, u + y) - 14, -252);
            float const h = scale2(hi, sh), lw = scale2(lo, sh);
            float const oh = __shfl_xor_sync(0xffffffffu, h, 1);
            float const ol = __shfl_xor_sync(0xffffffffu, lw, 1);
            if (row_on && 8 * blk + u < eds) mx = max(mx, __float_as_uint(h) & 0x7FFFFFFFu);
            out[y] = (row & 1) ? make_float4(oh, ol, h, lw) : make_float4(h, lw, oh, ol);
          }
          // the even lane of a row pair (Re) stores the natural layout, the odd one
          // (Im) the transposed, two entries of its row at once
          int const j = 8 * blk + u;
          if (store && j < eds) {
            if (row & 1) {
              store_pair(dst + j, out);
            } else {
              dst[eds * j] = out[0];
              dst[eds * (j + 1)] = out[1];
            }
          }
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) atomicMax(g.slot_bits + slot, mx);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols)
                 : "memory");
  }
}

template <int kPad>
cudaError_t launch_steps(StepArgs const &args, cudaStream_t stream) {
  cudaError_t const e = cudaFuncSetAttribute(product_step_kernel<kPad>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(step_smem(kPad)));
  if (e != cudaSuccess) return e;
  product_step_kernel<kPad><<<static_cast<unsigned>(persistent_grid(args.n_units)), kStepThreads,
                              step_smem(kPad), stream>>>(args);
  return cudaGetLastError();
}

}  // namespace

int64_t prod_tc_a_bytes(int32_t eds) {
  return static_cast<int64_t>(prod_tc_pad(eds) / (kTK / 2)) * kStageA;
}

cudaError_t products_tc(float4 *slots_n, float4 *slots_t, uint8_t *scratch, int64_t r_off,
                        int32_t *expo, int64_t r_expo, ProdGroup const *groups, int64_t n_groups,
                        int32_t const *r_slots, int64_t n_r, int32_t const *u_list,
                        int32_t const *out_tab, ProdTile const *tiles, int64_t n_tiles,
                        int32_t eds, unsigned int *slot_bits, int *err, cudaStream_t stream) {
  if (n_tiles == 0) return cudaSuccess;
  if (!prod_tc_supported(eds) || n_groups > 0x7fffffffLL || n_r > 0x7fffffffLL ||
      n_tiles > 0x7fffffffLL)
    return cudaErrorInvalidValue;
  int64_t const a_bytes = prod_tc_a_bytes(eds);
  prod_slice_a_kernel<<<static_cast<unsigned>(n_groups), kPSliceThreads, 0, stream>>>(
      scratch, expo, groups, slots_t, eds, a_bytes);
  if (n_r > 0)
    prod_slice_r_kernel<<<static_cast<unsigned>(n_r), kPSliceThreads, 0, stream>>>(
        scratch + r_off, expo + r_expo, r_slots, slots_n, eds);
  if (prod_tc_steps(eds)) {
    cudaError_t const se = cudaGetLastError();
    if (se != cudaSuccess) return se;
    StepArgs const args{scratch, a_bytes, r_off, tiles, static_cast<int32_t>(n_tiles), u_list,
                        expo, r_expo, out_tab, slots_n, slots_t, slot_bits, err, eds};
    return prod_tc_pad(eds) == 32 ? launch_steps<32>(args, stream)
                                  : launch_steps<16>(args, stream);
  }
  cudaError_t e = cudaFuncSetAttribute(product_gemm_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(kSmemBytes));
  if (e != cudaSuccess) return e;
  ProdTiles const tl{scratch, a_bytes, r_off, tiles, groups, u_list, eds, eds / (kTK / 2)};
  product_gemm_kernel<<<static_cast<unsigned>(persistent_grid(n_tiles)), kThreads, kSmemBytes,
                        stream>>>(tl, static_cast<int32_t>(n_tiles), expo, r_expo, out_tab,
                                  slots_n, slots_t, slot_bits, err);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace slaph
