// Weight preparation on the device: the fixed-order, shared-curvature pruner with joint INT8
// rounding that produces the `qweight` / `scales` the packer consumes
// (reference: sdacc/diffusion_research/reconstruction.py:55-133, `compress`).
//
// Output rows are independent and all share one curvature factor, so a column block is processed
// by four lanes per row: the row's slice lives in shared memory next to the block's factor tile,
// the lanes walk the groups in order (selection at the group's start, then rounding, error and
// update column by column inside the group, then the group's errors on the columns still open) and
// the errors of the block are applied to all later columns by an fp32 GEMM with a fixed summation
// order.  Every floating-point result is that of a separately rounded IEEE operation in the order
// the reference's tensor expressions apply them (the GEMM accumulates with fused multiply-adds in
// increasing k), which the CPU oracle repeats.
#include "ss_common.cuh"

namespace ss {
namespace {

constexpr int kLanesPerRow = 4;
constexpr int kRowsPerWarp = 32 / kLanesPerRow;
constexpr int kObsMaxRows = 64;      // rows a CTA walks at a time, at most
constexpr int kObsMaxWidth = 225;    // widest column block

// a / b, correctly rounded, from y = RN(1 / b): two residual corrections of the product a * y.  The
// first makes the quotient faithful, after which the second gives the rounded one (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990; needs b, y, the
// quotient and the residuals to stay clear of overflow and underflow, which the callers' ranges see to).
__device__ __forceinline__ float quotient(float a, float b, float y) {
  float q = __fmul_rn(a, y);
  q = __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
  return __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
}

__device__ __forceinline__ float round_to_grid(float v, float s) {
  // torch.round(v / s).clamp(-128, 127): round half to even
  return fminf(127.f, fmaxf(-128.f, rintf(__fdiv_rn(v, s))));
}

// Ranges in which quotient() is exact: divisors 2^-15 .. 2^15 (their squares 2^-30 .. 2^30), positive scales
// 2^-60 .. 2^60 (the rounded quotient takes the dividend's sign), dividends +0 and 2^-90 .. 2^60.  Outside
// (and for NaN) the IEEE division runs.
__device__ __forceinline__ bool within(float v, float lo, float hi) { return fabsf(v) >= lo && fabsf(v) <= hi; }
__device__ __forceinline__ bool dividend_ok(float v) {
  const uint32_t bits = __float_as_uint(v), lo = (127u - 90u) << 23, hi = (127u + 60u) << 23;
  return bits == 0u || (bits & 0x7fffffffu) - lo <= hi - lo;
}

// The columns of one group while it is walked: values (which become the finalised ones) and errors.
template <int G>
struct ObsGroup {
  float v[G], e[G], loss;
  unsigned mask;
};

// Walks a group: the two smallest scores (one or none in an incomplete group, ties to the lower column)
// are selected, then column by column it is rounded, its error taken and the group's later columns
// updated.  FAST takes complete groups only, divides by the reciprocals and returns whether every division
// was within their range: straight code without a branch, so that the loads of all columns go out first.
template <int G, bool JOINT, bool FAST>
__device__ __forceinline__ bool walk_group(ObsGroup<G>& g, int i0, int span, const float* const (&row)[G], const float* recip,
                                           const float* square, const float* square_recip, float s, float s_recip,
                                           float v_limit) {
  bool ok = true;
  if constexpr (FAST) span = G;
  const int remove = max(0, 2 - (G - span));
  float low = 0.f, next = 0.f;
  int first = 0, second = 0;
#pragma unroll
  for (int c = 0; c < G; ++c) {
    if (c < span) {
      const float vv = __fmul_rn(g.v[c], g.v[c]);
      float score;
      if constexpr (FAST) {
        score = quotient(vv, square[c], square_recip[c]);
        ok = ok && dividend_ok(vv);
      } else {
        score = __fdiv_rn(vv, square[c]);
      }
      if (c == 0) {
        low = score;
      } else if (score < low) {
        next = low; second = first; low = score; first = c;
      } else if (c == 1 || score < next) {
        next = score; second = c;
      }
    }
  }
  g.mask = (remove > 0 ? 1u << first : 0u) | (remove > 1 ? 1u << second : 0u);
#pragma unroll
  for (int c = 0; c < G; ++c) {
    g.e[c] = 0.f;
    if (c < span) {
      float frow[G];                                   // frow[o] = factor[i0 + c][i0 + o] for o >= c
#pragma unroll
      for (int o = c & ~1; o < G; o += 2) {
        const float2 f = *reinterpret_cast<const float2*>(row[c] + i0 + o);
        frow[o] = f.x;
        frow[o + 1] = f.y;
      }
      float fin = g.v[c];
      if constexpr (JOINT && FAST) {
        const float q = fminf(127.f, fmaxf(-128.f, copysignf(rintf(quotient(g.v[c], s, s_recip)), g.v[c])));
        ok = ok && fabsf(g.v[c]) <= v_limit;
        fin = __fmul_rn(q, s);
      } else if constexpr (JOINT) {
        fin = __fmul_rn(round_to_grid(g.v[c], s), s);
      }
      if (g.mask >> c & 1u) fin = 0.f;
      const float d = __fsub_rn(g.v[c], fin);
      if constexpr (FAST) {
        g.e[c] = quotient(d, frow[c], recip[c]);
        ok = ok && dividend_ok(d);
      } else {
        g.e[c] = __fdiv_rn(d, frow[c]);
      }
      g.loss = __fadd_rn(g.loss, __fmul_rn(__fmul_rn(g.e[c], g.e[c]), 0.5f));
      g.v[c] = fin;
#pragma unroll
      for (int o = c + 1; o < G; ++o) g.v[o] = __fsub_rn(g.v[o], __fmul_rn(g.e[c], frow[o]));
    }
  }
  return ok;
}

__host__ __device__ __forceinline__ int obs_pitch(int width) {
  // floats between two rows' open values: 16 (mod 32), so that the 16-byte accesses of two rows'
  // lanes fall into different banks
  return (width + 47) / 32 * 32 - 16;
}
// Factor tile: the upper triangle row after row, row i from column i rounded down to 4 up to the
// width rounded up to 4.  This is where column j of row i lies, less j.
__host__ __device__ __forceinline__ int obs_row(int i, int width) {
  const int wp = (width + 3) & ~3, a = i >> 2;
  return 4 * a * wp - 8 * a * (a - 1) + (i & 3) * (wp - 4 * a) - 4 * a;
}
__host__ __device__ __forceinline__ int obs_tile_floats(int width) { return obs_row(width, width) + (width & ~3); }

// The same with IEEE divisions, out of line: the straight code of the fast form has to stay small, the
// warps of a CTA run it in different places and out of the instruction caches otherwise.
template <int G, bool JOINT>
__device__ __noinline__ void walk_group_ieee(ObsGroup<G>* g, int i0, int span, const float* tile, int width, const float* square,
                                             float s) {
  const float* row[G];
#pragma unroll
  for (int c = 0; c < G; ++c) row[c] = tile + obs_row(i0 + c, width);
  walk_group<G, JOINT, false>(*g, i0, span, row, nullptr, square + i0, nullptr, s, 0.f, 0.f);
}

// One column block [start, start+width).  Bound by the dependent chain of a column.  All four lanes of
// a row walk it together in registers, a group at a time (the reciprocals of the divisors are made
// once, which turns a division into five dependent multiply-adds), and they share the update of the
// columns still open, group by group, 16 bytes at a time in the packed form of two.  Eight lanes per row,
// a division in each step of the chain and an update of all open columns per column: 161 us per block of
// 192 columns, 9216 rows; four lanes and groups with the IEEE division inline 101 us; out of line 86 us;
// complete groups in code without branches 74 us.
// Shared memory: factor tile, three reciprocal rows, then per row two float rows (open values, which
// become the finalised ones, and errors), then a byte per group and row (its selected zeros).
template <int G, bool JOINT>
__global__ void __launch_bounds__(kObsMaxRows * kLanesPerRow, 1)
obs_block_kernel(float* __restrict__ w, int rows, int64_t columns, int64_t start, int width, int rows_per_cta,
                 const float* __restrict__ upper, const float* __restrict__ scales, float minus_zero,
                 uint8_t* __restrict__ zeros, float* __restrict__ errors, float* __restrict__ losses) {
  extern __shared__ __align__(16) unsigned char smem[];
  float* tile = reinterpret_cast<float*>(smem);
  const int wp = (width + 3) & ~3, pitch = obs_pitch(width), groups = (width + G - 1) / G;
  float* recip = tile + obs_tile_floats(width);              // of the diagonal
  float* square = recip + wp;                                // diagonal squared, and its reciprocal
  float* square_recip = square + wp;
  float* open_all = square_recip + wp;
  float* err_all = open_all + rows_per_cta * pitch;
  uint8_t* chosen_all = reinterpret_cast<uint8_t*>(err_all + rows_per_cta * pitch);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sl = lane & (kLanesPerRow - 1);
  const int slot = threadIdx.x / kLanesPerRow, warps = blockDim.x >> 5;

  for (int r = warp; r < width; r += warps) {
    float* dst = tile + obs_row(r, width);
    const float* src = upper + (start + r) * columns + start;
    for (int c = (r & ~3) + lane; c < wp; c += 32) {
      if (c < width) ptx::cp_async4(dst + c, src + c); else dst[c] = 0.f;
    }
  }
  ptx::cp_async_wait_all();
  __syncthreads();
  bool in_range = true;
  for (int i = threadIdx.x; i < width; i += blockDim.x) {
    const float d = tile[obs_row(i, width) + i], dd = __fmul_rn(d, d);
    recip[i] = __fdiv_rn(1.f, d);
    square[i] = dd;
    square_recip[i] = __fdiv_rn(1.f, dd);
    in_range = in_range && within(d, 0x1p-15f, 0x1p15f);
  }
  const bool exact = __syncthreads_and(in_range);
  float* open = open_all + slot * pitch;
  float* err = err_all + slot * pitch;
  uint8_t* chosen = chosen_all + slot * groups;

  for (int base = blockIdx.x * rows_per_cta; base < rows; base += gridDim.x * rows_per_cta) {
    const int row = base + slot, warp_row = base + warp * kRowsPerWarp;
    // the warp's rows, one after the other, 128 bytes at a time, all in flight together
    for (int r = 0; r < kRowsPerWarp; ++r) {
      const float* wr = w + static_cast<int64_t>(warp_row + r) * columns + start;
      float* to = open_all + (warp * kRowsPerWarp + r) * pitch;
      for (int j = lane; j < wp; j += 32) {
        if (warp_row + r < rows && j < width) ptx::cp_async4(to + j, wr + j); else to[j] = 0.f;
      }
    }
    const float s = row < rows ? scales[row] : 1.f;
    const float s_recip = __fdiv_rn(1.f, s);
    const float v_limit = s >= 0x1p-60f && s <= 0x1p60f ? 0x1p60f : -1.f;
    float loss = row < rows ? losses[row] : 0.f;
    ptx::cp_async_wait_all();
    __syncwarp();
    for (int group = 0; group < groups; ++group) {
      const int i0 = group * G, span = min(G, width - i0);
      const float* frow[G];
#pragma unroll
      for (int c = 0; c < G; ++c) frow[c] = tile + obs_row(i0 + c, width);
      ObsGroup<G> g;
#pragma unroll
      for (int c = 0; c < G; ++c) g.v[c] = c < span ? open[i0 + c] : 0.f;
      g.loss = loss;
      bool ok = exact && span == G;
      if (ok) ok = walk_group<G, JOINT, true>(g, i0, span, frow, recip + i0, square + i0, square_recip + i0, s, s_recip, v_limit);
      if (!ok) {
        ObsGroup<G> again;
#pragma unroll
        for (int c = 0; c < G; ++c) again.v[c] = c < span ? open[i0 + c] : 0.f;
        again.loss = loss;
        walk_group_ieee<G, JOINT>(&again, i0, span, tile, width, square, s);
        g = again;
      }
      loss = g.loss;
      // The group's errors on the open columns: o = (o - e0 f0) - e1 f1 ..., two columns at a time.  The
      // packed multiply and add of sm_100a are contracted to one rounding whatever their rounding
      // modifiers say, so the product is made by a multiply-add onto a -0 that the compiler does not know
      // (the same value, sign of zero included).
      const float2 none = make_float2(minus_zero, minus_zero);
      const int i1 = i0 + G;
      if (i1 < width) {
        float2 minus[G];
#pragma unroll
        for (int c = 0; c < G; ++c) minus[c] = make_float2(-g.e[c], -g.e[c]);
        if (G == 6 && (i1 & 2) && sl == 0) {
          float2 o = *reinterpret_cast<float2*>(open + i1);
#pragma unroll
          for (int c = 0; c < G; ++c)
            o = __fadd2_rn(o, __ffma2_rn(minus[c], *reinterpret_cast<const float2*>(frow[c] + i1), none));
          *reinterpret_cast<float2*>(open + i1) = o;
        }
        // two quads a step, so that one's chain hides the other's
        for (int j = ((i1 + 3) & ~3) + 4 * sl; j < width; j += 8 * kLanesPerRow) {
          const int jb = j + 4 * kLanesPerRow < width ? j + 4 * kLanesPerRow : j;
          const float4 oa = *reinterpret_cast<const float4*>(open + j), ob = *reinterpret_cast<const float4*>(open + jb);
          float2 o[4] = {make_float2(oa.x, oa.y), make_float2(oa.z, oa.w), make_float2(ob.x, ob.y), make_float2(ob.z, ob.w)};
#pragma unroll
          for (int c = 0; c < G; ++c) {
            const float4 fa = *reinterpret_cast<const float4*>(frow[c] + j), fb = *reinterpret_cast<const float4*>(frow[c] + jb);
            o[0] = __fadd2_rn(o[0], __ffma2_rn(minus[c], make_float2(fa.x, fa.y), none));
            o[1] = __fadd2_rn(o[1], __ffma2_rn(minus[c], make_float2(fa.z, fa.w), none));
            o[2] = __fadd2_rn(o[2], __ffma2_rn(minus[c], make_float2(fb.x, fb.y), none));
            o[3] = __fadd2_rn(o[3], __ffma2_rn(minus[c], make_float2(fb.z, fb.w), none));
          }
          *reinterpret_cast<float4*>(open + jb) = make_float4(o[2].x, o[2].y, o[3].x, o[3].y);
          *reinterpret_cast<float4*>(open + j) = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
        }
      }
      __syncwarp();                   // every lane of the row has read the group's values
#pragma unroll
      for (int c = 0; c < G; ++c)
        if (sl == (c & (kLanesPerRow - 1)) && c < span) { open[i0 + c] = g.v[c]; err[i0 + c] = g.e[c]; }
      if (sl == 0) chosen[group] = static_cast<uint8_t>(g.mask);
      __syncwarp();
    }
    if (sl == 0 && row < rows) losses[row] = loss;
    for (int r = 0; r < kRowsPerWarp && warp_row + r < rows; ++r) {
      const int at = warp * kRowsPerWarp + r;
      const int64_t out = static_cast<int64_t>(warp_row + r) * columns + start;
      float* er = errors + static_cast<int64_t>(warp_row + r) * width;
      for (int j = lane; j < width; j += 32) {
        w[out + j] = open_all[at * pitch + j];
        er[j] = err_all[at * pitch + j];
        zeros[out + j] = chosen_all[at * groups + j / G] >> (j % G) & 1u;
      }
    }
    __syncwarp();
  }
}

// w[r, stop + j] -= sum_k errors[r, k] * upper[start + k, stop + j], the sum taken as
// acc = fma(e, u, acc) from acc = 0 in increasing k.  Bound by the FP32 pipes and, next to them, the
// shared-memory port: 128 x 96 output tile (blocks are 192 wide), 8 x 12 per thread (rows ty*4+i and 64+ty*4+i,
// columns 32*h+tx*4+j) in the packed form of two multiply-adds, so that five 16-byte reads feed 48 of them.  Two
// slabs: the next one's B comes in by asynchronous copies, its A through registers, while the current one
// is multiplied.  VEC: 16-byte accesses of the factor, the errors and w (all rows 16-byte aligned).
// 8 x 8 per thread, scalar multiply-adds, scalar loads, one slab: 202 us a block (26 TFLOP/s) at 9216 x
// 3072 in blocks of 192; packed multiply-adds and two slabs alone 174 us; 8 x 16 per thread
// on 128 x 128 tiles, two CTAs per SM, 148 us; this form, three CTAs per SM, 130 us.
// (Half a slab of A in registers, 128 x 64 tiles with four CTAs: 133 us; two CTAs of this tile: 140 us.)
constexpr int kTileM = 128, kTileN = 96, kTileK = 16, kQuads = kTileN / 32;

template <bool VEC>
__global__ void __launch_bounds__(128, 3)
obs_trailing_kernel(float* __restrict__ w, int rows, int64_t columns, int64_t start, int width,
                    const float* __restrict__ upper, const float* __restrict__ errors) {
  __shared__ __align__(16) float a_s[2][kTileK][kTileM];
  __shared__ __align__(16) float b_s[2][kTileK][kTileN];
  const int64_t stop = start + width;
  const int cols = static_cast<int>(columns - stop);
  const int row0 = blockIdx.y * kTileM, col0 = blockIdx.x * kTileN;
  const int t = threadIdx.x, tx = t & 7, ty = t >> 3;
  // this thread's share of a slab: the 16 k of one row of A, 16 columns of one k of B
  const float* a_src = errors + static_cast<int64_t>(row0 + t) * width;
  const bool a_ok = row0 + t < rows;
  float a_reg[kTileK];
  auto fetch_a = [&](int k0) {
#pragma unroll
    for (int i = 0; i < kTileK; i += 4) {
      if constexpr (VEC) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (a_ok && k0 + i < width) v = *reinterpret_cast<const float4*>(a_src + k0 + i);
        a_reg[i] = v.x; a_reg[i + 1] = v.y; a_reg[i + 2] = v.z; a_reg[i + 3] = v.w;
      } else {
#pragma unroll
        for (int j = i; j < i + 4; ++j) a_reg[j] = a_ok && k0 + j < width ? a_src[k0 + j] : 0.f;
      }
    }
  };
  auto store_a = [&](int slab) {
#pragma unroll
    for (int i = 0; i < kTileK; ++i) a_s[slab][i][t] = a_reg[i];
  };
  auto fetch_b = [&](int k0, int slab) {
    const bool k_ok = k0 + ty < width;
    const float* src = upper + (start + (k_ok ? k0 + ty : 0)) * columns + stop;
#pragma unroll
    for (int h = 0; h < kQuads; ++h)
#pragma unroll
      for (int j = 0; j < 4; j += VEC ? 4 : 1) {
        const int c = 32 * h + tx * 4 + j;
        const bool in = k_ok && col0 + c < cols;                   // VEC: cols is a multiple of four
        const float* from = src + (in ? col0 + c : 0);
        if constexpr (VEC) ptx::cp_async16(&b_s[slab][ty][c], from, in ? 16u : 0u);
        else ptx::cp_async4(&b_s[slab][ty][c], from, in ? 4u : 0u);
      }
  };
  float2 acc[8][2 * kQuads];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 2 * kQuads; ++j) acc[i][j] = make_float2(0.f, 0.f);
  fetch_a(0);
  fetch_b(0, 0);
  store_a(0);
  ptx::cp_async_wait_all();
  __syncthreads();
  int slab = 0;
  for (int k0 = 0; k0 < width; k0 += kTileK, slab ^= 1) {
    const bool more = k0 + kTileK < width;
    if (more) { fetch_b(k0 + kTileK, slab ^ 1); fetch_a(k0 + kTileK); }
#pragma unroll
    for (int k = 0; k < kTileK; ++k) {
      float2 b[2 * kQuads];
#pragma unroll
      for (int h = 0; h < kQuads; ++h) {
        const float4 v = *reinterpret_cast<const float4*>(&b_s[slab][k][32 * h + tx * 4]);
        b[2 * h] = make_float2(v.x, v.y);
        b[2 * h + 1] = make_float2(v.z, v.w);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 v = *reinterpret_cast<const float4*>(&a_s[slab][k][64 * h + ty * 4]);
        const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 2 * kQuads; ++j) acc[4 * h + i][j] = __ffma2_rn(make_float2(a[i], a[i]), b[j], acc[4 * h + i][j]);
      }
    }
    if (more) {
      store_a(slab ^ 1);
      ptx::cp_async_wait_all();
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = row0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4);
    if (r >= rows) continue;
    float* wr = w + static_cast<int64_t>(r) * columns + stop;
#pragma unroll
    for (int h = 0; h < kQuads; ++h) {
      const int c = col0 + 32 * h + tx * 4;
      const float2 lo = acc[i][2 * h], hi = acc[i][2 * h + 1];
      if constexpr (VEC) {
        if (c < cols) {
          float4 v = *reinterpret_cast<float4*>(wr + c);
          v = make_float4(__fsub_rn(v.x, lo.x), __fsub_rn(v.y, lo.y), __fsub_rn(v.z, hi.x), __fsub_rn(v.w, hi.y));
          *reinterpret_cast<float4*>(wr + c) = v;
        }
      } else {
        const float sum[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (c + j < cols) wr[c + j] = __fsub_rn(wr[c + j], sum[j]);
      }
    }
  }
}

// Final export: q = clamp(rint(w / scale)) with the selected zeros forced to 0; status bit 0 is set
// when q * scale differs from w (checked only when check_grid), bit 1 when a complete group holds
// more than group - 2 nonzeros, bit 2 when w holds a non-finite value.  Bound by HBM: a CTA per row, a
// thread per group, two columns at a time where the rows allow it (PAIRS).  One thread per group over the
// whole weight, its row found by a 64-bit division: 91 us at 9216 x 3072 (4:6); now 43 us.
template <int G, bool PAIRS>
__global__ void __launch_bounds__(256)
obs_finish_kernel(const float* __restrict__ w, const float* __restrict__ scales, const uint8_t* __restrict__ zeros,
                  int64_t columns, int check_grid, int8_t* __restrict__ q, int32_t* __restrict__ status) {
  const int64_t row = blockIdx.x;
  const float s = scales[row];
  w += row * columns;
  zeros += row * columns;
  q += row * columns;
  int flags = 0;
  for (int64_t c0 = static_cast<int64_t>(threadIdx.x) * G; c0 < columns; c0 += static_cast<int64_t>(blockDim.x) * G) {
    const int span = static_cast<int>(columns - c0 < G ? columns - c0 : G);
    int nonzero = 0;
    auto column = [&](float v, bool zero) {
      const int value = zero ? 0 : static_cast<int>(round_to_grid(v, s));
      nonzero += value != 0;
      if (check_grid && !(__fmul_rn(static_cast<float>(value), s) == v)) flags |= 1;
      if (!isfinite(v)) flags |= 4;
      return static_cast<char>(value);
    };
#pragma unroll
    for (int c = 0; c < G; c += PAIRS ? 2 : 1) {
      if (c < span) {
        if constexpr (PAIRS) {
          const float2 v = *reinterpret_cast<const float2*>(w + c0 + c);
          const uchar2 z = *reinterpret_cast<const uchar2*>(zeros + c0 + c);
          *reinterpret_cast<char2*>(q + c0 + c) = make_char2(column(v.x, z.x), column(v.y, z.y));
        } else {
          q[c0 + c] = column(w[c0 + c], zeros[c0 + c]);
        }
      }
    }
    if (span == G && nonzero > G - 2) flags |= 2;
  }
  if (flags) atomicOr(status, flags);
}

}  // namespace
}  // namespace ss

using namespace ss;

static size_t obs_block_smem(int width, int group, int rows) {
  const int wp = (width + 3) & ~3;
  return (static_cast<size_t>(obs_tile_floats(width)) + 3 * wp + 2 * rows * obs_pitch(width)) * sizeof(float) +
         static_cast<size_t>(rows) * ((width + group - 1) / group);
}

extern "C" int ss_obs_max_blocksize(void) { return kObsMaxWidth; }

extern "C" int ss_obs_block(float* w, int64_t rows, int64_t columns, int64_t start, int64_t width,
                            const float* upper, const float* scales, int group, int joint,
                            uint8_t* zeros, float* errors, float* losses, void* stream) {
  SS_REQUIRE(w && upper && scales && zeros && errors && losses, SS_E_ARG, "obs_block: null pointer");
  SS_REQUIRE(mode_ok(group), SS_E_ARG, "obs_block: group must be 4, 6 or 8");
  SS_REQUIRE(rows > 0 && rows < (1ll << 31) && columns > 0 && columns < (1ll << 31), SS_E_ARG, "obs_block: invalid shape");
  SS_REQUIRE(start >= 0 && width > 0 && start + width <= columns && start % group == 0, SS_E_ARG,
             "obs_block: the block [start, start+width) must lie inside the row and start on a group boundary");
  SS_REQUIRE(width <= kObsMaxWidth, SS_E_ARG, "obs_block: a block of %lld columns does not fit shared memory (limit %d)",
             static_cast<long long>(width), kObsMaxWidth);
  int device = 0, sms = 0;
  SS_CUDA(cudaGetDevice(&device));
  SS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  // spread the rows over all SMs, whole warps of eight; the widest blocks leave room for 56 rows
  int64_t per_cta = ((rows + sms - 1) / sms + kRowsPerWarp - 1) / kRowsPerWarp * kRowsPerWarp;
  if (per_cta > kObsMaxRows) per_cta = kObsMaxRows;
  const int wide = static_cast<int>(width);
  while (obs_block_smem(wide, group, static_cast<int>(per_cta)) > 227 * 1024) per_cta -= kRowsPerWarp;
  const size_t smem = obs_block_smem(wide, group, static_cast<int>(per_cta));
  const int64_t wanted = (rows + per_cta - 1) / per_cta;
  const unsigned grid = static_cast<unsigned>(wanted < sms ? wanted : sms);
  auto kernel = group == 4 ? (joint ? obs_block_kernel<4, true> : obs_block_kernel<4, false>)
              : group == 6 ? (joint ? obs_block_kernel<6, true> : obs_block_kernel<6, false>)
                           : (joint ? obs_block_kernel<8, true> : obs_block_kernel<8, false>);
  SS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  kernel<<<grid, static_cast<unsigned>(per_cta) * kLanesPerRow, smem, static_cast<cudaStream_t>(stream)>>>(
      w, static_cast<int>(rows), columns, start, wide, static_cast<int>(per_cta), upper, scales, -0.0f, zeros,
      errors, losses);
  SS_CUDA(cudaGetLastError());
  return SS_OK;
}

extern "C" int ss_obs_trailing(float* w, int64_t rows, int64_t columns, int64_t start, int64_t width,
                               const float* upper, const float* errors, void* stream) {
  SS_REQUIRE(w && upper && errors, SS_E_ARG, "obs_trailing: null pointer");
  SS_REQUIRE(rows > 0 && rows < (1ll << 31) && columns > 0 && columns < (1ll << 31), SS_E_ARG, "obs_trailing: invalid shape");
  SS_REQUIRE(start >= 0 && width > 0 && start + width <= columns, SS_E_ARG, "obs_trailing: block outside the row");
  const int64_t cols = columns - start - width;
  if (cols == 0) return SS_OK;
  const dim3 grid(static_cast<unsigned>((cols + kTileN - 1) / kTileN), static_cast<unsigned>((rows + kTileM - 1) / kTileM));
  SS_REQUIRE(grid.y <= 65535, SS_E_ARG, "obs_trailing: too many rows for one launch");
  const bool vec = ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(upper) | reinterpret_cast<uintptr_t>(errors)) & 15) == 0 &&
                   columns % 4 == 0 && width % 4 == 0 && start % 4 == 0;
  auto kernel = vec ? obs_trailing_kernel<true> : obs_trailing_kernel<false>;
  kernel<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(
      w, static_cast<int>(rows), columns, start, static_cast<int>(width), upper, errors);
  SS_CUDA(cudaGetLastError());
  return SS_OK;
}

extern "C" int ss_obs_finish(const float* w, const float* scales, const uint8_t* zeros, int64_t rows,
                             int64_t columns, int group, int check_grid, int8_t* qweight, int32_t* status,
                             void* stream) {
  SS_REQUIRE(w && scales && zeros && qweight && status, SS_E_ARG, "obs_finish: null pointer");
  SS_REQUIRE(mode_ok(group), SS_E_ARG, "obs_finish: group must be 4, 6 or 8");
  SS_REQUIRE(rows > 0 && rows < (1ll << 31) && columns > 0 && columns < (1ll << 31), SS_E_ARG, "obs_finish: invalid shape");
  const bool pairs = columns % 2 == 0 && (reinterpret_cast<uintptr_t>(w) & 7) == 0 &&
                     ((reinterpret_cast<uintptr_t>(zeros) | reinterpret_cast<uintptr_t>(qweight)) & 1) == 0;
  auto kernel = group == 4 ? (pairs ? obs_finish_kernel<4, true> : obs_finish_kernel<4, false>)
              : group == 6 ? (pairs ? obs_finish_kernel<6, true> : obs_finish_kernel<6, false>)
                           : (pairs ? obs_finish_kernel<8, true> : obs_finish_kernel<8, false>);
  const int64_t groups = (columns + group - 1) / group;
  const unsigned threads = groups >= 256 ? 256u : static_cast<unsigned>((groups + 31) / 32 * 32);
  kernel<<<static_cast<unsigned>(rows), threads, 0, static_cast<cudaStream_t>(stream)>>>(w, scales, zeros, columns, check_grid,
                                                                                       qweight, status);
  SS_CUDA(cudaGetLastError());
  return SS_OK;
}
