// Ladder search and row quantisation (hi2/encode.py:53-173, hi2/ladder_kernel.py:44-101).
//
// fit kernel   one thread per (row, block), two for blocks of 64.  The lanes of a warp take consecutive
//              ROWS of the same block, so the column weights d of the block are warp-uniform (staged
//              in shared memory) and the block's weights stay in registers for the whole grid search
//              and the least-squares refits.  The work is about 350 instructions per weight (effort
//              "normal") against 4 bytes read: bound by the fp32 pipe (70 % busy at blocks of 32).
// row kernel   one warp per row: row-wide extrema of (lo, step), the three fp16 row constants, the
//              parameter bytes, the decoded fp16 ladders, and optionally the nearest codes and the
//              weighted error of the row, in one pass over the row.  table_row_kernel does this for all
//              candidates of an error table at once, without codes.  Both are bound by instruction issue.
#include "common.cuh"

namespace hi2 {
namespace {

struct GridSpec {
  float v[8];
  int g;
  float one;  // 1.0, as a kernel argument
  float packed_from;  // steps above it take the packed arithmetic: 0, or infinity for more levels than it holds
};

// Block sums are formed in the order of torch's CPU reduction over a contiguous inner dimension
// (aten/src/ATen/native/cpu/SumKernel.cpp): the block is read as B/8 vectors of 8 lanes, four
// interleaved vector accumulators take vectors 0-3 and then 4-7, the accumulators are added left
// to right, and the 8 lanes of the result are added left to right.  The reference's (lo, step)
// depend on these sums to the last bit (the least-squares formulas cancel), so with this order
// the search returns the reference's ladders bit for bit; a plain left-to-right sum does not.
template <int B>
__device__ __forceinline__ float fold_lane(const float (&v)[B / 8]) {
  if constexpr (B == 16) {
    return v[0] + v[1];
  } else if constexpr (B == 32) {
    return ((v[0] + v[1]) + v[2]) + v[3];
  } else {
    return (((v[0] + v[4]) + (v[1] + v[5])) + (v[2] + v[6])) + (v[3] + v[7]);
  }
}

// Codes are rint((x - lo) / safe) with an IEEE division in the reference.  Here one correctly
// rounded reciprocal of `safe` serves the block and every quotient is finished with Markstein's
// fused correction, which yields the correctly rounded quotient itself, so rint sees the very number
// the division would give.  Steps outside the range the correction covers (rc.fast false: tiny, huge,
// or a significand of all ones), negative ones and ladders of more than 2^23 steps take true divisions.
//
// Everything else is done for two neighbouring columns per instruction (packed fp32 multiplies and
// fused multiply-adds), since the search is bound by instruction issue: 12 instructions a pair where
// the scalar form had 28.  A packed add would be contracted with the packed multiply that feeds it, and
// the sum of a separately rounded product is what the reference has; so additions are written as
// a * one + b with a `one` the compiler cannot see through, which rounds exactly like a + b.
// Signs are turned so that one constant serves all: the block is kept as -x, the differences as
// lo - x, never above zero (a code below zero becomes zero either way), and multiplied by -1 / step.
// Rounding to an integer is one addition of 2^23, and the product of the integer with the step comes
// out of the same fused multiply-add that takes the 2^23 off again (2^23 * step is exact).
constexpr float SHIFT = 8388608.0f;

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 add2(float2 a, float2 b, float2 one) { return __ffma2_rn(a, one, b); }
__device__ __forceinline__ float2 min2(float2 a, float b) { return make_float2(fminf(a.x, b), fminf(a.y, b)); }

// The columns one thread keeps, as pairs of -x.  Blocks of 16 and 32 belong to one thread: pair 4 j + 2 h + i
// holds columns 8 j + 4 h + 2 i and its right neighbour.  A block of 64 is shared by two neighbouring
// lanes (one thread's registers hold the values but not the differences, and the unrolled code of 64
// columns no longer fits the instruction cache): lane `half` keeps the columns with h = half, as pair
// 2 j + i.
template <int B>
struct Block {
  static constexpr bool SHARED = B == 64;
  static constexpr int PAIRS = SHARED ? 16 : B / 2;
  float2 nx[PAIRS];
};

// Column weights of a block: shared memory, or (tensors that read different inputs) global memory.
template <bool GROUPED>
__device__ __forceinline__ float4 weights4(const float* d) {
  if (GROUPED) return __ldg(reinterpret_cast<const float4*>(d));
  return *reinterpret_cast<const float4*>(d);
}

// One ladder prepared for the packed loop.
struct Step {
  float2 neg_r, safe, step, off;  // -1 / step, step, step, -2^23 step
  bool fast;
};
__device__ __forceinline__ Step make_step(float step, float packed_from) {
  Step s;
  const float safe = (step == 0.0f) ? 1.0f : step;
  const Recip rc = make_recip(safe);
  s.fast = rc.fast && safe > packed_from;
  s.neg_r = both(-rc.r), s.safe = both(safe), s.step = both(step), s.off = both(-SHIFT * step);
  return s;
}
// 2^23 + the code of two columns, an = min(lo - x, 0)
__device__ __forceinline__ float2 shifted_codes(float2 an, const Step& s, float top, float2 one) {
  const float2 q0 = __fmul2_rn(an, s.neg_r);
  const float2 q = __ffma2_rn(__ffma2_rn(q0, s.safe, an), s.neg_r, q0);
  return min2(add2(q, both(SHIFT), one), top);
}
// d * (x_hat - x)^2 of two columns
__device__ __forceinline__ float2 weighted_square(float2 an, float2 nx, float2 d, const Step& s, float2 lo, float top,
                                                  float2 one) {
  const float2 rec = add2(__ffma2_rn(shifted_codes(an, s, top, one), s.step, s.off), lo, one);
  const float2 diff = add2(rec, nx, one);
  return __fmul2_rn(d, __fmul2_rn(diff, diff));
}

// N sums over the block in the reference's order; v(j, h, first pair, t) gives the terms of the two pairs
// of one 128-bit load of the weights.  Lanes that share a block exchange the four partial sums of
// their half, so all lanes of the warp have to call this together.
template <int B, int N, typename F>
__device__ __forceinline__ void block_sums(float (&out)[N], int half, float2 one, F&& v) {
  if constexpr (Block<B>::SHARED) {
    float2 s[2][N];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 t[2][N], far[2][N];
      v(j, half, 2 * j, t);
      v(j + 4, half, 2 * (j + 4), far);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int k = 0; k < N; ++k) {
          t[i][k] = add2(t[i][k], far[i][k], one);
          s[i][k] = j == 0 ? t[i][k] : add2(s[i][k], t[i][k], one);
        }
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const float mine[4] = {s[0][k].x, s[0][k].y, s[1][k].x, s[1][k].y};
      float other[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) other[i] = __shfl_xor_sync(0xffffffffu, mine[i], 1);
      out[k] = half ? other[0] : mine[0];
#pragma unroll
      for (int i = 1; i < 4; ++i) out[k] = out[k] + (half ? other[i] : mine[i]);
#pragma unroll
      for (int i = 0; i < 4; ++i) out[k] = out[k] + (half ? mine[i] : other[i]);
    }
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float2 s[2][N];
#pragma unroll
      for (int j = 0; j < B / 8; ++j) {
        float2 t[2][N];
        v(j, h, 4 * j + 2 * h, t);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int k = 0; k < N; ++k) s[i][k] = j == 0 ? t[i][k] : add2(s[i][k], t[i][k], one);
      }
#pragma unroll
      for (int k = 0; k < N; ++k) {
        out[k] = h == 0 ? s[0][k].x : out[k] + s[0][k].x;
        out[k] = out[k] + s[0][k].y;
        out[k] = out[k] + s[1][k].x;
        out[k] = out[k] + s[1][k].y;
      }
    }
  }
}

// The error of one ladder with true divisions, for steps the packed loop does not cover.
template <int B>
__device__ __noinline__ float block_error_careful(const float* __restrict__ x, const float* d, float lo, float step,
                                                  float nmax) {
  const float safe = (step == 0.0f) ? 1.0f : step;
  float err = 0.0f;
#pragma unroll 1
  for (int l = 0; l < 8; ++l) {
    float v[B / 8];
#pragma unroll
    for (int j = 0; j < B / 8; ++j) {
      const int t = 8 * j + l;
      float q = rintf(__fdiv_rn(x[t] - lo, safe));
      q = fminf(fmaxf(q, 0.0f), nmax);
      const float diff = (lo + q * step) - x[t];
      v[j] = d[t] * (diff * diff);
    }
    const float s = fold_lane<B>(v);
    err = (l == 0) ? s : err + s;
  }
  return err;
}

// lo - x of a pair, never above zero
__device__ __forceinline__ float2 below(float2 nx, float2 lo, float2 one) { return min2(add2(nx, lo, one), 0.0f); }

// Error of one ladder.  `an` (HAVE_AN) holds the differences of this lo; x and d are the block's in
// memory.
template <int B, bool GROUPED, bool HAVE_AN>
__device__ __forceinline__ float block_error_exact(const Block<B>& blk, const float2* an, const float* __restrict__ x,
                                                   const float* d, int half, float lo, float step, float nmax, float2 one,
                                                   float packed_from) {
  const Step s = make_step(step, packed_from);
  const float2 lo2 = both(lo);
  const float top = SHIFT + nmax;
  float err[1];
  block_sums<B, 1>(err, half, one, [&](int j, int h, int p, float2 (&t)[2][1]) {
    const float4 dv = weights4<GROUPED>(d + 8 * j + 4 * h);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 a = HAVE_AN ? an[p + i] : below(blk.nx[p + i], lo2, one);
      t[i][0] = weighted_square(a, blk.nx[p + i], i == 0 ? make_float2(dv.x, dv.y) : make_float2(dv.z, dv.w), s, lo2, top, one);
    }
  });
  return s.fast ? err[0] : block_error_careful<B>(x, d, lo, step, nmax);
}

// The same with codes rint(num * (1 / step)), one instruction a pair instead of four, for ladders of at
// most 16 levels.  The product can round to another integer than the quotient only where the column
// lies within delta of the middle between two levels, that is where |x_hat - x| is within delta of
// step / 2: the two quotients differ by 2^-23 of at most nmax - 1/2, and num, q * step, lo + q * step and
// the difference were each rounded once, so delta = 2^-24 (5 nmax step + |lo|).  The squares the sum
// needs anyway are compared with step^2 / 4 (their own rounding is in the sixth nmax * step below); a
// block with such a column, about one in 500 warps and ladders at 4 levels and one in 100 at 16, is
// done again exactly.  At 256 levels it would be one in eight, and the exact form is used at once.
// 11008 x 4096, normal effort, 4 levels, blocks of 16 / 32 / 64, us: scalar form 914 / 862 / 973 us, packed
// 790 / 710 / 742, this 713 / 670 / 709.
template <int B, bool GROUPED>
__device__ __forceinline__ float block_error(const Block<B>& blk, const float2 (&an)[Block<B>::PAIRS],
                                             const float* __restrict__ x, const float* d, int half, float lo, float step,
                                             float nmax, float2 one, float packed_from) {
  bool sure = nmax <= 15.0f && step > 1e-15f && step < 1e15f;
  if (Block<B>::SHARED) sure = __all_sync(0xffffffffu, sure);
  if (sure) {
    const float2 lo2 = both(lo), neg_r = both(-__frcp_rn(step)), step2 = both(step), off = both(-SHIFT * step);
    const float2 neg_mid = both(-((0.5f * step) * (0.5f * step)));
    const float top = SHIFT + nmax;
    float near = INFINITY;
    float err[1];
    block_sums<B, 1>(err, half, one, [&](int j, int h, int p, float2 (&t)[2][1]) {
      const float4 dv = weights4<GROUPED>(d + 8 * j + 4 * h);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 c = min2(__ffma2_rn(an[p + i], neg_r, both(SHIFT)), top);
        const float2 diff = add2(add2(__ffma2_rn(c, step2, off), lo2, one), blk.nx[p + i], one);
        const float2 sq = __fmul2_rn(diff, diff);
        const float2 mid = add2(sq, neg_mid, one);
        near = fminf(fminf(near, fabsf(mid.x)), fabsf(mid.y));
        t[i][0] = __fmul2_rn(i == 0 ? make_float2(dv.x, dv.y) : make_float2(dv.z, dv.w), sq);
      }
    });
    sure = near > 6.3e-8f * step * (6.0f * nmax * step + fabsf(lo));
    if (Block<B>::SHARED) sure = __all_sync(0xffffffffu, sure);
    if (sure) return err[0];
  }
  return block_error_exact<B, GROUPED, true>(blk, an, x, d, half, lo, step, nmax, one, packed_from);
}

// Sum over the block of d * (distance beyond `edge`)^2, on the side where lo - x > 0 (LOW) or < 0: what the
// columns that a ladder ending at `edge` clips contribute to its error.  In any order: it serves as a
// bound.
template <int B, bool GROUPED, bool LOW>
__device__ __forceinline__ float clipped_error(const Block<B>& blk, const float* d, int half, float edge, float2 one) {
  const float2 e2 = both(edge);
  float2 sum[2] = {both(0.0f), both(0.0f)};
#pragma unroll
  for (int g = 0; g < Block<B>::PAIRS / 2; ++g) {
    const float4 dv = weights4<GROUPED>(d + (Block<B>::SHARED ? 8 * g + 4 * half : 4 * g));
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float2 m = add2(blk.nx[2 * g + i], e2, one);
      m = LOW ? make_float2(fmaxf(m.x, 0.0f), fmaxf(m.y, 0.0f)) : min2(m, 0.0f);
      sum[i] = __ffma2_rn(__fmul2_rn(m, m), i == 0 ? make_float2(dv.x, dv.y) : make_float2(dv.z, dv.w), sum[i]);
    }
  }
  float s = (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
  if (Block<B>::SHARED) s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}

constexpr int FIT_THREADS = 128, FIT_WARPS = FIT_THREADS / 32;

struct FitShared {
  __align__(16) float d[FIT_WARPS][64];
  float high_error[8][FIT_THREADS];  // a thread's own, by grid point
};

// The ladders of one tile: 32 rows (16 for blocks of 64) of FIT_WARPS blocks, a block per warp.
template <int B, bool GROUPED, bool BOUND>
__device__ __forceinline__ void fit_tile(FitShared& shared, int64_t row_tile, int64_t blk_tile, const float* __restrict__ w,
                                         int64_t ldw, const float* __restrict__ d_all, const int32_t* __restrict__ row_d,
                                         int64_t n_rows, int64_t nb, const GridSpec& grid, int refits, float nmax,
                                         float* __restrict__ lo_out, float* __restrict__ st_out,
                                         float* __restrict__ err_out) {
  constexpr bool SHARED = Block<B>::SHARED;
  constexpr int PAIRS = Block<B>::PAIRS, ROWS = SHARED ? 16 : 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = SHARED ? lane & 1 : 0;
  const int64_t blk = blk_tile * FIT_WARPS + warp;
  if (blk >= nb) return;  // uniform over the warp
  const int64_t row = row_tile * ROWS + (SHARED ? lane >> 1 : lane);
  const bool live = row < n_rows;
  const int64_t row_c = live ? row : n_rows - 1;
  const float* src = w + row_c * ldw + blk * B;
  const float2 one = both(grid.one);
  // GROUPED: d is [groups, k] and row r is weighted by d[row_d[r]] (tensors that read different
  // inputs, e.g. the experts of a layer, searched in one launch)
  const float* d;
  if (GROUPED) {
    d = d_all + (int64_t)row_d[row_c] * (nb * B) + blk * B;
  } else {
    // one weight per lane: hi2_ladder_grid's weights may start at any float
    for (int t = lane; t < B; t += 32) shared.d[warp][t] = __ldg(d_all + blk * B + t);
    __syncwarp();
    d = shared.d[warp];
  }

  Block<B> r;
  float mn = 0.0f, mx = 0.0f;
#pragma unroll
  for (int q = 0; q < PAIRS / 2; ++q) {
    const float4 v = *reinterpret_cast<const float4*>(src + (SHARED ? 8 * q + 4 * half : 4 * q));
    if (q == 0) mn = v.x, mx = v.x;
    mn = fminf(fminf(fminf(fminf(mn, v.x), v.y), v.z), v.w), mx = fmaxf(fmaxf(fmaxf(fmaxf(mx, v.x), v.y), v.z), v.w);
    r.nx[2 * q] = make_float2(-v.x, -v.y), r.nx[2 * q + 1] = make_float2(-v.z, -v.w);
  }
  if (SHARED) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
  }
  const float span = mx - mn;
  const Recip rc_n = make_recip(nmax);  // nmax is 3, 15 or 255: div_by is the IEEE quotient

  // BOUND: a grid point clips the columns outside [lo, hi], hi = mx - v span, and they alone cost it the clipped
  // errors at both ends.  Where those exceed the best error so far the point cannot win and is passed
  // over: with 16 levels or more the steps are so fine that few grid points survive.  The codes of these
  // columns are 0 and the highest; hi is moved out by 1e-6 of the block's range, more than the
  // roundings that lie between it and the highest level, and 1e-4 covers those of the sums.
  bool weights_ok = true;
  const bool bound = BOUND && grid.g > 1;  // a single point has nothing to be measured against
  if (bound) {
    const float slack = 1e-6f * (fabsf(mn) + fabsf(mx));
    float lowest = 0.0f;
#pragma unroll
    for (int g = 0; g < PAIRS / 2; ++g) {
      const float4 dv = weights4<GROUPED>(d + (SHARED ? 8 * g + 4 * half : 4 * g));
      lowest = fminf(lowest, fminf(fminf(dv.x, dv.y), fminf(dv.z, dv.w)));
    }
    if (SHARED) lowest = fminf(lowest, __shfl_xor_sync(0xffffffffu, lowest, 1));
    weights_ok = lowest >= 0.0f;
#pragma unroll 1
    for (int gj = 0; gj < grid.g; ++gj)
      shared.high_error[gj][threadIdx.x] =
          grid.v[gj] == 0.0f ? 0.0f : clipped_error<B, GROUPED, false>(r, d, half, (mx - grid.v[gj] * span) + slack, one);
  }

  float best_lo = 0.0f, best_st = 0.0f, best_err = 0.0f;
#pragma unroll 1
  for (int gi = 0; gi < grid.g; ++gi) {
    const float lo = mn + grid.v[gi] * span;
    float2 an[PAIRS];
#pragma unroll
    for (int p = 0; p < PAIRS; ++p) an[p] = below(r.nx[p], both(lo), one);
    float low_error = 0.0f;
    if (bound && grid.v[gi] != 0.0f) low_error = clipped_error<B, GROUPED, true>(r, d, half, lo, one);
#pragma unroll 1
    for (int gj = 0; gj < grid.g; ++gj) {
      const float step = div_by((mx - grid.v[gj] * span) - lo, nmax, rc_n);
      if (bound && (gi | gj) != 0) {
        bool beaten = weights_ok && step > 1e-15f && 0.9999f * (low_error + shared.high_error[gj][threadIdx.x]) > best_err;
        if (SHARED) beaten = __all_sync(0xffffffffu, beaten);
        if (beaten) continue;
      }
      const float err = block_error<B, GROUPED>(r, an, src, d, half, lo, step, nmax, one, grid.packed_from);
      if ((gi | gj) == 0 || err < best_err) best_lo = lo, best_st = step, best_err = err;
    }
  }

#pragma unroll 1
  for (int it = 0; it < refits; ++it) {
    // sums over the block of d, d c, d c^2, -d x, -d c x and -x, c the code
    float sums[6];
    const Step s = make_step(best_st, grid.packed_from);
    const float2 lo2 = both(best_lo);
    const float top = SHIFT + nmax, safe = s.safe.x;
    block_sums<B, 6>(sums, half, one, [&](int j, int h, int p, float2 (&t)[2][6]) {
      const float4 dv = weights4<GROUPED>(d + 8 * j + 4 * h);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 nx = r.nx[p + i], dp = i == 0 ? make_float2(dv.x, dv.y) : make_float2(dv.z, dv.w);
        float2 c;
        if (s.fast) {
          c = add2(shifted_codes(below(nx, lo2, one), s, top, one), both(-SHIFT), one);
        } else {
          c.x = fminf(fmaxf(rintf(__fdiv_rn(-nx.x - best_lo, safe)), 0.0f), nmax);
          c.y = fminf(fmaxf(rintf(__fdiv_rn(-nx.y - best_lo, safe)), 0.0f), nmax);
        }
        const float2 dc = __fmul2_rn(dp, c);
        t[i][0] = dp, t[i][1] = dc, t[i][2] = __fmul2_rn(dc, c), t[i][3] = __fmul2_rn(dp, nx);
        t[i][4] = __fmul2_rn(dc, nx), t[i][5] = nx;
      }
    });
    const float sd = sums[0], sc = sums[1], scc = sums[2], sw = -sums[3], scw = -sums[4], sum = -sums[5];
    const float det = sd * scc - sc * sc;
    const bool ok = fabsf(det) > 1e-20f;
    const float step = ok ? __fdiv_rn(sd * scw - sc * sw, det) : 0.0f;
    const float lo = ok ? __fdiv_rn(sw - step * sc, fmaxf(sd, 1e-20f)) : __fdiv_rn(sum, (float)B);
    const float err = block_error_exact<B, GROUPED, false>(r, nullptr, src, d, half, lo, step, nmax, one, grid.packed_from);
    if (err < best_err && step > 0.0f) best_lo = lo, best_st = step, best_err = err;
  }

  if (live && half == 0) {
    const int64_t o = row * nb + blk;
    lo_out[o] = best_lo;
    st_out[o] = best_st;
    if (err_out != nullptr) err_out[o] = best_err;
  }
}

template <int B, bool GROUPED, bool BOUND>
__global__ void __launch_bounds__(FIT_THREADS, (B == 16 ? 5 : 4))
fit_kernel(const float* __restrict__ w, int64_t ldw, const float* __restrict__ d_all,
           const int32_t* __restrict__ row_d, int64_t n_rows, int64_t nb, GridSpec grid, int refits, float nmax, float* __restrict__ lo_out,
           float* __restrict__ st_out, float* __restrict__ err_out) {
  __shared__ FitShared shared;
  const int64_t blk_tile = (int64_t)blockIdx.z * gridDim.y + blockIdx.y;  // one dimension ends at 65535
  fit_tile<B, GROUPED, BOUND>(shared, blockIdx.x, blk_tile, w, ldw, d_all, row_d, n_rows, nb, grid, refits, nmax, lo_out,
                              st_out, err_out);
}

// Every candidate (levels, block) of an error table in one launch: the tiles of one candidate after the
// other along the grid, so the last wave of one is filled by the next.
constexpr int TABLE_MAX = 16;
struct TableCandidate {
  float *lo, *st;
  float nmax;
  int block, bound;
  unsigned row_tiles, first_tile;
};
struct TableSpec {
  TableCandidate c[TABLE_MAX];
  int n;
};

template <bool GROUPED>
__global__ void __launch_bounds__(FIT_THREADS, 4)
table_fit_kernel(const float* __restrict__ w, int64_t ldw, const float* __restrict__ d_all,
                 const int32_t* __restrict__ row_d, int64_t n_rows, int64_t k, const __grid_constant__ GridSpec grid,
                 int refits, const __grid_constant__ TableSpec table) {
  __shared__ FitShared shared;
  int at = 0;
  while (at + 1 < table.n && blockIdx.x >= table.c[at + 1].first_tile) ++at;
  const TableCandidate& c = table.c[at];
  const unsigned tile = blockIdx.x - c.first_tile;
  const int64_t row_tile = tile % c.row_tiles, blk_tile = tile / c.row_tiles;
#define HI2_TILE(BB, CC)                                                                                              \
  fit_tile<BB, GROUPED, CC>(shared, row_tile, blk_tile, w, ldw, d_all, row_d, n_rows, k / BB, grid, refits, c.nmax, c.lo, \
                            c.st, nullptr)
  if (c.block == 16) {
    if (c.bound) HI2_TILE(16, true);
    else HI2_TILE(16, false);
  } else if (c.block == 32) {
    if (c.bound) HI2_TILE(32, true);
    else HI2_TILE(32, false);
  } else {
    if (c.bound) HI2_TILE(64, true);
    else HI2_TILE(64, false);
  }
#undef HI2_TILE
}

// The grid as the kernels take it; *clips: every point moves an end of the ladder inwards, by half the
// range at most.
GridSpec make_grid(const float* grid_host, int g, float nmax, bool* clips) {
  GridSpec spec;
  spec.g = g, spec.one = 1.0f;
  spec.packed_from = nmax <= SHIFT ? 0.0f : INFINITY;  // 2^23 + a larger code is not a whole number
  *clips = true;
  for (int i = 0; i < 8; ++i) {
    spec.v[i] = i < g ? grid_host[i] : 0.0f;
    *clips = *clips && spec.v[i] >= 0.0f && spec.v[i] <= 0.5f;
  }
  return spec;
}

int launch_fit(const float* w, int64_t ldw, const float* d, const int32_t* row_d, const float* grid_host, int g,
               int refits, int n, int64_t n_rows, int64_t nb, int block, float* lo, float* st,
               float* err, cudaStream_t stream) {
  bool clips;
  const float nmax = (float)(n - 1);
  const GridSpec spec = make_grid(grid_host, g, nmax, &clips);
  const int64_t blk_tiles = ceil_div(nb, (int64_t)FIT_WARPS), layers = ceil_div(blk_tiles, (int64_t)65535);
  dim3 grid((unsigned)ceil_div(n_rows, block == 64 ? 16 : 32), (unsigned)ceil_div(blk_tiles, layers), (unsigned)layers);
  // Passing over grid points that their clipped columns rule out: 11008 x 4096, normal effort, blocks of 16 /
  // 32 / 64, us: 16 levels 682 / 645 / 682 -> 483 / 502 / 590, 256 levels 770 / 739 / 780 -> 360 / 295 / 301;
  // at 4 levels next to nothing is ruled out and the bounds cost 6 %.
  const bool bound = n >= 16 && clips;
#define HI2_FIT_V(BB, GG, CC)                                                                                       \
  fit_kernel<BB, GG, CC><<<grid, FIT_THREADS, 0, stream>>>(w, ldw, d, row_d, n_rows, nb, spec, refits, nmax, lo, st, err)
#define HI2_FIT(BB)                                     \
  do {                                                  \
    if (row_d != nullptr && bound) HI2_FIT_V(BB, true, true);    \
    else if (row_d != nullptr) HI2_FIT_V(BB, true, false);       \
    else if (bound) HI2_FIT_V(BB, false, true);                  \
    else HI2_FIT_V(BB, false, false);                            \
  } while (0)
  if (block == 16) HI2_FIT(16);
  if (block == 32) HI2_FIT(32);
  if (block == 64) HI2_FIT(64);
#undef HI2_FIT
#undef HI2_FIT_V
  return check_launch("fit_ladder");
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The three fp16 constants of a row from the extrema of its ladders (hi2/encode.py:95-119).
struct RowConstants {
  __half lm_h, ls_h, ss_h;
  float lm, ls, ss;
};
__device__ __forceinline__ RowConstants row_constants(float mxst, float mnlo, float mxlo) {
  RowConstants c;
  c.ss_h = __float2half_rn(__fdiv_rn(mxst, 255.0f)), c.ss = __half2float(c.ss_h);
  c.lm_h = __float2half_rn(mnlo), c.lm = __half2float(c.lm_h);
  float spread = mxlo - c.lm;
  spread = spread < 0.0f ? 0.0f : spread;
  c.ls_h = __float2half_rn(__fdiv_rn(spread, 255.0f)), c.ls = __half2float(c.ls_h);
  return c;
}
// Parameter bytes of one block against the rounded constants, and the ladder they decode to.
__device__ __forceinline__ void quantise_block(const RowConstants& c, float lo, float st, uint8_t& lu8, uint8_t& su8,
                                               float& lod, float& std_) {
  const float s = st < 0.0f ? 0.0f : st;
  float su = 0.0f, lu = 0.0f;
  if (c.ss > 0.0f) su = clamp_keep_nan(rintf(__fdiv_rn(s, fmaxf(c.ss, 1e-30f))), 0.0f, 255.0f);
  if (c.ls > 0.0f) lu = clamp_keep_nan(rintf(__fdiv_rn(lo - c.lm, fmaxf(c.ls, 1e-30f))), 0.0f, 255.0f);
  su8 = (uint8_t)su, lu8 = (uint8_t)lu;
  lod = round_f16(fmaf((float)lu8, c.ls, c.lm));
  std_ = round_f16((float)su8 * c.ss);
}

constexpr int ROW_THREADS = 256;
constexpr int ROW_WARPS = ROW_THREADS / 32;
constexpr int ROW_UN = 4;  // quads a lane loads before it computes
// Shared memory a row pass may ask for.  A kernel's limit is set to this and never to what one call needs: it
// is one setting for all threads of the process, and a thread that lowered it between another's setting and
// launch made that launch fail.
constexpr int ROW_SMEM_MAX = 200 * 1024;

// One WARP per row: the row-wide extrema, the constants and the parameter bytes need only warp
// shuffles, so no thread block barrier sits between the phases of a row and 64 rows are in flight
// per SM.  Dynamic shared memory: per warp the decoded lo[nb], step[nb] of its row.
// CODES / ENERGY: whether code bytes are written and the row energy is summed.  The ladders of the column
// loop ask for neither, and a pass over the weights is bound by instruction issue (73 % of the issue slots
// at a third of the copy bandwidth), so the instructions of unused outputs are compiled out.
template <int B, bool CODES, bool ENERGY>
__global__ void __launch_bounds__(ROW_THREADS, 4)
row_kernel(const float* __restrict__ lo_in, const float* __restrict__ st_in,
           const float* __restrict__ w, int64_t ldw, const float* __restrict__ d_all,
           const int32_t* __restrict__ row_d, float nmax, int64_t n_rows, int64_t k, uint8_t* __restrict__ params, uint16_t* __restrict__ consts,
           float* __restrict__ lo_d, float* __restrict__ st_d, int64_t ldp,
           uint8_t* __restrict__ codes, float* __restrict__ sse, float* __restrict__ energy) {
  extern __shared__ float dyn[];
  const int64_t nb = k / B;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* s_lo = dyn + (size_t)warp * 2 * nb;
  float* s_st = s_lo + nb;

  for (int64_t row = (int64_t)blockIdx.x * ROW_WARPS + warp; row < n_rows; row += (int64_t)gridDim.x * ROW_WARPS) {
    const float* lo_r = lo_in + row * nb;
    const float* st_r = st_in + row * nb;
    // ---- row-wide extrema -----------------------------------------------------------------
    float mxst = -INFINITY, mnlo = INFINITY, mxlo = -INFINITY;
    for (int64_t b = lane; b < nb; b += 32) {
      const float s = st_r[b], l = lo_r[b];
      mxst = fmaxf(mxst, s < 0.0f ? 0.0f : s);
      mnlo = fminf(mnlo, l);
      mxlo = fmaxf(mxlo, l);
    }
    mxst = warp_max(mxst), mnlo = warp_min(mnlo), mxlo = warp_max(mxlo);
    // ---- the three fp16 row constants -------------------------------------------------------
    const RowConstants rc = row_constants(mxst, mnlo, mxlo);
    if (lane == 0 && consts != nullptr) {
      consts[row * 3 + 0] = __half_as_ushort(rc.lm_h);
      consts[row * 3 + 1] = __half_as_ushort(rc.ls_h);
      consts[row * 3 + 2] = __half_as_ushort(rc.ss_h);
    }
    // ---- parameter bytes and decoded ladders ------------------------------------------------
    __syncwarp();  // the previous row's readers of s_lo / s_st are done
    for (int64_t b = lane; b < nb; b += 32) {
      uint8_t lu8, su8;
      float lod, std_;
      quantise_block(rc, lo_r[b], st_r[b], lu8, su8, lod, std_);
      s_lo[b] = lod;
      s_st[b] = std_;
      if (params != nullptr) {
        params[(row * nb + b) * 2 + 0] = lu8;
        params[(row * nb + b) * 2 + 1] = su8;
      }
      if (lo_d != nullptr) lo_d[row * ldp + b] = lod;
      if (st_d != nullptr) st_d[row * ldp + b] = std_;
    }
    if (sse == nullptr && codes == nullptr && energy == nullptr) continue;
    __syncwarp();
    // ---- nearest codes, weighted error, energy ------------------------------------------------
    // A lane takes ROW_UN quads per trip, all loads first, to keep enough bytes in flight.  Codes are
    // rint((w - lo) / step) with an IEEE division in the reference; the quotient is formed with the
    // block's correctly rounded reciprocal and Markstein's fused correction, which gives the same
    // correctly rounded number.
    const float* wr = w + row * ldw;
    const float* d = d_all + (row_d != nullptr ? (int64_t)row_d[row] * k : 0);  // the row's own column weights
    float acc = 0.0f, en = 0.0f;
    for (int64_t j0 = (int64_t)lane * 4; j0 < k; j0 += 128 * ROW_UN) {
      float4 wq[ROW_UN], dq[ROW_UN];
#pragma unroll
      for (int u = 0; u < ROW_UN; ++u) {
        const int64_t j = j0 + u * 128;
        if (j < k) {
          wq[u] = *reinterpret_cast<const float4*>(wr + j);
          dq[u] = *reinterpret_cast<const float4*>(d + j);
        }
      }
#pragma unroll
      for (int u = 0; u < ROW_UN; ++u) {
        const int64_t j = j0 + u * 128;
        if (j >= k) break;
        const int64_t b = j / B;
        const float lod = s_lo[b], std_ = s_st[b];
        const float safe = (std_ == 0.0f) ? 1.0f : std_;
        const Recip rc = make_recip(safe);
        const float ws[4] = {wq[u].x, wq[u].y, wq[u].z, wq[u].w}, ds[4] = {dq[u].x, dq[u].y, dq[u].z, dq[u].w};
        uint8_t cs[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float num = ws[t] - lod;
          float c;
          if (rc.fast) {
            const float q0 = num * rc.r;
            c = rintf(fmaf(fmaf(-q0, safe, num), rc.r, q0));
          } else {
            c = rintf(__fdiv_rn(num, safe));
          }
          if (std_ == 0.0f) c = 0.0f;
          c = clamp_keep_nan(c, 0.0f, nmax);
          const float diff = round_f16(lod + c * std_) - ws[t];
          acc += ds[t] * (diff * diff);
          if (ENERGY) en += ds[t] * (ws[t] * ws[t]);
          if (CODES) cs[t] = (uint8_t)c;
        }
        if (CODES) *reinterpret_cast<uchar4*>(codes + row * k + j) = make_uchar4(cs[0], cs[1], cs[2], cs[3]);
      }
    }
    acc = warp_sum(acc);
    if (ENERGY) en = warp_sum(en);
    if (lane == 0) {
      if (sse != nullptr) sse[row] = acc;
      if (ENERGY) energy[row] = en;
    }
  }
}

// The row pass of an error table: what row_kernel does for one candidate without codes, for all of them
// with one pass over the row.  Per candidate the warp forms the row constants and keeps the decoded
// ladders in shared memory as (lo, step) in fp16, which they are, and the step's reciprocal; then every
// 128-bit load of the row and of the weights serves all candidates, two columns per instruction as in
// the search above.  Each lane sums its columns in row_kernel's order, so the errors are the same bits.
// Bound by instruction issue.  Six candidates, one pass each -> this: 11008 x 4096 400 -> 216 us, 1024 x 2048
// 53 -> 22.
struct TableEntry {
  __half2 ladder;
  float r;  // 1 / step; 0 for step == 0 (the code is 0), NaN where the quotient has to be a true division
};

// d (x_hat - x)^2 of four columns, added in column order.
__device__ __forceinline__ float table_quad(const float4 w, const float4 d, const TableEntry e, float nmax, float2 one,
                                            float acc) {
  const float2 ladder = __half22float2(e.ladder);
  const float2 lo2 = both(ladder.x), st2 = both(ladder.y), neg_r = both(-e.r), off = both(-SHIFT * ladder.y);
  const float top = SHIFT + nmax;
  float2 v[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float2 nx = i == 0 ? make_float2(-w.x, -w.y) : make_float2(-w.z, -w.w);
    const float2 an = below(nx, lo2, one);
    const float2 q0 = __fmul2_rn(an, neg_r);
    const float2 q = __ffma2_rn(__ffma2_rn(q0, st2, an), neg_r, q0);
    const float2 c = min2(add2(q, both(SHIFT), one), top);
    const float2 sum = add2(__ffma2_rn(c, st2, off), lo2, one);
    const float2 diff = add2(__half22float2(__float22half2_rn(sum)), nx, one);
    v[i] = __fmul2_rn(i == 0 ? make_float2(d.x, d.y) : make_float2(d.z, d.w), __fmul2_rn(diff, diff));
  }
  return (((acc + v[0].x) + v[0].y) + v[1].x) + v[1].y;
}
// The same with true divisions, for entries without a usable reciprocal.
__device__ __noinline__ float table_quad_careful(const float4 w, const float4 d, const TableEntry e, float nmax, float acc) {
  const float lod = __low2float(e.ladder), step = __high2float(e.ladder);
  const float ws[4] = {w.x, w.y, w.z, w.w}, ds[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    float c = rintf(__fdiv_rn(ws[t] - lod, step == 0.0f ? 1.0f : step));
    if (step == 0.0f) c = 0.0f;
    c = clamp_keep_nan(c, 0.0f, nmax);
    const float diff = round_f16(lod + c * step) - ws[t];
    acc += ds[t] * (diff * diff);
  }
  return acc;
}

constexpr int TABLE_ROW_WARPS = 4;
template <int N>  // candidates [first, first + N)
__global__ void __launch_bounds__(TABLE_ROW_WARPS * 32)
table_row_kernel(const float* __restrict__ w, int64_t ldw, const float* __restrict__ d_all,
                 const int32_t* __restrict__ row_d, int64_t n_rows, int64_t k, const __grid_constant__ TableSpec table,
                 int first, int entries, float one_arg, float* __restrict__ sse, float* __restrict__ energy) {
  extern __shared__ __align__(16) TableEntry table_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  TableEntry* own = table_smem + (size_t)warp * entries;
  const float2 one = both(one_arg);
  int shift[N];
  float nmax[N];
  const TableEntry* ladders[N];
  {
    int off = 0;
#pragma unroll
    for (int c = 0; c < N; ++c) {
      shift[c] = table.c[first + c].block == 16 ? 4 : table.c[first + c].block == 32 ? 5 : 6;
      nmax[c] = table.c[first + c].nmax;
      ladders[c] = own + off;
      off += (int)(k >> shift[c]);
    }
  }
  for (int64_t row = (int64_t)blockIdx.x * TABLE_ROW_WARPS + warp; row < n_rows; row += (int64_t)gridDim.x * TABLE_ROW_WARPS) {
    __syncwarp();  // the previous row's readers are done
    int off = 0;
    for (int c = first; c < first + N; ++c) {
      const int nb = (int)(k / table.c[c].block);
      const float* lo_r = table.c[c].lo + row * nb;
      const float* st_r = table.c[c].st + row * nb;
      float mxst = -INFINITY, mnlo = INFINITY, mxlo = -INFINITY;
      for (int b = lane; b < nb; b += 32) {
        const float s = st_r[b], l = lo_r[b];
        mxst = fmaxf(mxst, s < 0.0f ? 0.0f : s);
        mnlo = fminf(mnlo, l);
        mxlo = fmaxf(mxlo, l);
      }
      mxst = warp_max(mxst), mnlo = warp_min(mnlo), mxlo = warp_max(mxlo);
      const RowConstants rc = row_constants(mxst, mnlo, mxlo);
      for (int b = lane; b < nb; b += 32) {
        uint8_t lu8, su8;
        float lod, std_;
        quantise_block(rc, lo_r[b], st_r[b], lu8, su8, lod, std_);
        const Recip r = make_recip(std_);
        TableEntry e;
        e.ladder = __halves2half2(__float2half_rn(lod), __float2half_rn(std_));
        e.r = std_ == 0.0f ? 0.0f : (r.fast ? r.r : __int_as_float(0x7fc00000));
        own[off + b] = e;
      }
      off += nb;
    }
    __syncwarp();
    const float* wr = w + row * ldw;
    const float* d = d_all + (row_d != nullptr ? (int64_t)row_d[row] * k : 0);
    float acc[N], en = 0.0f;
#pragma unroll
    for (int c = 0; c < N; ++c) acc[c] = 0.0f;
    for (int64_t j0 = (int64_t)lane * 4; j0 < k; j0 += 128 * ROW_UN) {
      float4 wq[ROW_UN], dq[ROW_UN];
#pragma unroll
      for (int u = 0; u < ROW_UN; ++u) {
        const int64_t j = j0 + u * 128;
        if (j < k) {
          wq[u] = *reinterpret_cast<const float4*>(wr + j);
          dq[u] = *reinterpret_cast<const float4*>(d + j);
        }
      }
#pragma unroll 1
      for (int u = 0; u < ROW_UN; ++u) {
        const int j = (int)j0 + u * 128;
        if (j >= k) break;
        const float4 wv = u == 0 ? wq[0] : u == 1 ? wq[1] : u == 2 ? wq[2] : wq[3];
        const float4 dv = u == 0 ? dq[0] : u == 1 ? dq[1] : u == 2 ? dq[2] : dq[3];
        if (energy != nullptr) {
          en += dv.x * (wv.x * wv.x);
          en += dv.y * (wv.y * wv.y);
          en += dv.z * (wv.z * wv.z);
          en += dv.w * (wv.w * wv.w);
        }
        TableEntry e[N];
        bool usable = true;
#pragma unroll
        for (int c = 0; c < N; ++c) e[c] = ladders[c][j >> shift[c]], usable = usable && e[c].r == e[c].r;
        if (usable) {
#pragma unroll
          for (int c = 0; c < N; ++c) acc[c] = table_quad(wv, dv, e[c], nmax[c], one, acc[c]);
        } else {
#pragma unroll
          for (int c = 0; c < N; ++c) acc[c] = table_quad_careful(wv, dv, e[c], nmax[c], acc[c]);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const float a = warp_sum(acc[c]);
      if (lane == 0) sse[(int64_t)(first + c) * n_rows + row] = a;
    }
    if (energy != nullptr) {
      en = warp_sum(en);
      if (lane == 0) energy[row] = en;
    }
  }
}

// sse of given codes against given decoded ladders (the tail of the GPTQ path).
template <int B>
__global__ void __launch_bounds__(ROW_THREADS)
sse_kernel(const uint8_t* __restrict__ codes, const float* __restrict__ w, int64_t ldw,
           const float* __restrict__ d, const float* __restrict__ lo, const float* __restrict__ st,
           int64_t ldp, int64_t n_rows, int64_t k, float* __restrict__ sse) {
  __shared__ float red[ROW_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int64_t row = blockIdx.x; row < n_rows; row += gridDim.x) {
    float acc = 0.0f;
    for (int64_t j = (int64_t)tid * 4; j < k; j += ROW_THREADS * 4) {
      const float4 wv = *reinterpret_cast<const float4*>(w + row * ldw + j);
      const float4 dv = *reinterpret_cast<const float4*>(d + j);
      const uchar4 cv = *reinterpret_cast<const uchar4*>(codes + row * k + j);
      const float lod = lo[row * ldp + j / B], std_ = st[row * ldp + j / B];
      const float ws[4] = {wv.x, wv.y, wv.z, wv.w}, ds[4] = {dv.x, dv.y, dv.z, dv.w};
      const float cs[4] = {(float)cv.x, (float)cv.y, (float)cv.z, (float)cv.w};
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float diff = round_f16(lod + cs[t] * std_) - ws[t];
        acc += ds[t] * (diff * diff);
      }
    }
    acc = warp_sum(acc);
    __syncthreads();
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (tid == 0) {
      float a = 0.0f;
#pragma unroll
      for (int i = 0; i < ROW_THREADS / 32; ++i) a += red[i];
      sse[row] = a;
    }
  }
}

bool block_ok(int block) { return block == 16 || block == 32 || block == 64; }

}  // namespace
}  // namespace hi2

extern "C" int hi2_ladder_grid(const float* wb, const float* db, const float* grid_host, int g,
                               int n, int64_t n_rows, int64_t nb, int block, float* lo,
                               float* step, float* err, void* stream) {
  using namespace hi2;
  HI2_REQUIRE(block_ok(block), "ladder_grid: block must be 16, 32 or 64");
  HI2_REQUIRE(g >= 1 && g <= 8 && grid_host, "ladder_grid: the grid has 1 to 8 points");
  HI2_REQUIRE(n >= 2, "ladder_grid: n must be at least 2");
  if (n_rows == 0 || nb == 0) return HI2_OK;
  HI2_REQUIRE(wb && db && lo && step, "ladder_grid: null pointer");
  HI2_REQUIRE(aligned16(wb), "ladder_grid: wb must be 16-byte aligned");
  return launch_fit(wb, nb * block, db, nullptr, grid_host, g, 0, n, n_rows, nb, block, lo, step, err,
                    static_cast<cudaStream_t>(stream));
}

extern "C" int hi2_fit_ladder_grouped(const float* w, int64_t ldw, const float* d, const int32_t* row_d,
                                      const float* grid_host, int g, int refits, int n, int64_t n_rows,
                                      int64_t k, int block, float* lo, float* step, void* stream) {
  using namespace hi2;
  HI2_REQUIRE(block_ok(block), "fit_ladder: block must be 16, 32 or 64");
  HI2_REQUIRE(k > 0 && k % block == 0, "fit_ladder: k must be a multiple of the block");
  HI2_REQUIRE(g >= 1 && g <= 8 && grid_host, "fit_ladder: the grid has 1 to 8 points");
  HI2_REQUIRE(n >= 2 && refits >= 0, "fit_ladder: bad n or refits");
  if (n_rows == 0) return HI2_OK;
  HI2_REQUIRE(w && d && lo && step, "fit_ladder: null pointer");
  HI2_REQUIRE(aligned16(w) && aligned16(d) && ldw % 4 == 0 && ldw >= k, "fit_ladder: w, d alignment or ldw");
  return launch_fit(w, ldw, d, row_d, grid_host, g, refits, n, n_rows, k / block, block, lo, step,
                    nullptr, static_cast<cudaStream_t>(stream));
}

extern "C" int hi2_fit_ladder(const float* w, int64_t ldw, const float* d, const float* grid_host,
                              int g, int refits, int n, int64_t n_rows, int64_t k, int block,
                              float* lo, float* step, void* stream) {
  return hi2_fit_ladder_grouped(w, ldw, d, nullptr, grid_host, g, refits, n, n_rows, k, block, lo, step, stream);
}

extern "C" int hi2_quantize_rows_grouped(const float* lo, const float* step, const float* w, int64_t ldw,
                                         const float* d, const int32_t* row_d, int nbits, int64_t n_rows,
                                         int64_t k, int block, uint8_t* params, uint16_t* consts, float* lo_d,
                                         float* step_d, int64_t ldp, uint8_t* codes, float* sse,
                                         float* energy, void* stream) {
  using namespace hi2;
  HI2_REQUIRE(block_ok(block), "quantize_rows: block must be 16, 32 or 64");
  HI2_REQUIRE(k > 0 && k % block == 0, "quantize_rows: k must be a multiple of the block");
  HI2_REQUIRE(nbits >= 1 && nbits <= 8, "quantize_rows: nbits out of range");
  if (n_rows == 0) return HI2_OK;
  HI2_REQUIRE(lo && step, "quantize_rows: null ladders");
  const bool scan = codes || sse || energy;
  if (scan) {
    HI2_REQUIRE(w && d, "quantize_rows: codes, sse and energy need w and d");
    HI2_REQUIRE(aligned16(w) && aligned16(d) && ldw % 4 == 0 && ldw >= k,
                "quantize_rows: w, d alignment or ldw");
    HI2_REQUIRE(codes == nullptr || (reinterpret_cast<uintptr_t>(codes) & 3u) == 0,
                "quantize_rows: codes must be 4-byte aligned");
  }
  HI2_REQUIRE((lo_d == nullptr && step_d == nullptr) || ldp >= k / block, "quantize_rows: ldp");
  const int64_t nb = k / block;
  const size_t smem = (size_t)ROW_WARPS * (2 * nb) * sizeof(float);
  HI2_REQUIRE(smem <= (size_t)ROW_SMEM_MAX, "quantize_rows: k too large for the ladder cache");
  const int64_t want = ceil_div(n_rows, (int64_t)ROW_WARPS);
  const unsigned grid = (unsigned)(want < 148 * 8 ? want : 148 * 8);
  const float nmax = (float)((1 << nbits) - 1);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
#define HI2_ROW_V(BB, CC, EE)                                                                              \
  do {                                                                                                     \
    if (smem > 48 * 1024 &&                                                                                \
        cudaFuncSetAttribute(row_kernel<BB, CC, EE>, cudaFuncAttributeMaxDynamicSharedMemorySize,          \
                             ROW_SMEM_MAX) != cudaSuccess)                                                 \
      return fail(HI2_ERR_LAUNCH, "quantize_rows: cannot reserve shared memory");                          \
    row_kernel<BB, CC, EE><<<grid, ROW_THREADS, smem, s>>>(lo, step, w, ldw, d, row_d, nmax, n_rows, k,      \
                                                           params, consts, lo_d, step_d, ldp, codes, sse,    \
                                                           energy);                                          \
  } while (0)
#define HI2_ROW(BB)                                     \
  do {                                                  \
    if (codes != nullptr && energy != nullptr) HI2_ROW_V(BB, true, true);   \
    else if (codes != nullptr) HI2_ROW_V(BB, true, false);                  \
    else if (energy != nullptr) HI2_ROW_V(BB, false, true);                 \
    else HI2_ROW_V(BB, false, false);                                       \
  } while (0)
  if (block == 16) HI2_ROW(16);
  if (block == 32) HI2_ROW(32);
  if (block == 64) HI2_ROW(64);
#undef HI2_ROW
#undef HI2_ROW_V
  return check_launch("quantize_rows");
}

extern "C" int hi2_quantize_rows(const float* lo, const float* step, const float* w, int64_t ldw,
                                 const float* d, int nbits, int64_t n_rows, int64_t k, int block,
                                 uint8_t* params, uint16_t* consts, float* lo_d, float* step_d,
                                 int64_t ldp, uint8_t* codes, float* sse, float* energy,
                                 void* stream) {
  return hi2_quantize_rows_grouped(lo, step, w, ldw, d, nullptr, nbits, n_rows, k, block, params, consts, lo_d, step_d,
                                   ldp, codes, sse, energy, stream);
}

extern "C" int hi2_error_table(const float* w, int64_t ldw, const float* d, const int32_t* row_d, const float* grid_host,
                               int g, int refits, int n_cand, const int32_t* nbits_host, const int32_t* block_host,
                               int64_t n_rows, int64_t k, float* lo, float* step, float* sse, float* energy, void* stream) {
  using namespace hi2;
  HI2_REQUIRE(n_cand >= 1 && n_cand <= TABLE_MAX && nbits_host && block_host, "error_table: one to 16 candidates");
  HI2_REQUIRE(g >= 1 && g <= 8 && grid_host, "fit_ladder: the grid has 1 to 8 points");
  HI2_REQUIRE(refits >= 0, "fit_ladder: bad n or refits");
  for (int c = 0; c < n_cand; ++c) {
    HI2_REQUIRE(block_ok(block_host[c]), "fit_ladder: block must be 16, 32 or 64");
    HI2_REQUIRE(k > 0 && k % block_host[c] == 0, "fit_ladder: k must be a multiple of the block");
    HI2_REQUIRE(nbits_host[c] >= 1 && nbits_host[c] <= 8, "quantize_rows: nbits out of range");
    HI2_REQUIRE(ROW_WARPS * 2 * (k / block_host[c]) * (int64_t)sizeof(float) <= ROW_SMEM_MAX,
                "quantize_rows: k too large for the ladder cache");  // the limit of the one-candidate pass
  }
  if (n_rows == 0) return HI2_OK;
  HI2_REQUIRE(w && d && lo && step && sse, "fit_ladder: null pointer");
  HI2_REQUIRE(aligned16(w) && aligned16(d) && ldw % 4 == 0 && ldw >= k, "fit_ladder: w, d alignment or ldw");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  bool clips;
  const GridSpec spec = make_grid(grid_host, g, 255.0f, &clips);  // 8 bits at most
  TableSpec table;
  table.n = n_cand;
  int64_t tiles = 0, offset = 0;
  for (int c = 0; c < n_cand; ++c) {
    TableCandidate& x = table.c[c];
    const int64_t nb = k / block_host[c], row_tiles = ceil_div(n_rows, block_host[c] == 64 ? 16 : 32);
    x.block = block_host[c], x.nmax = (float)((1 << nbits_host[c]) - 1);
    x.bound = nbits_host[c] >= 4 && clips;
    x.lo = lo + offset, x.st = step + offset;
    x.row_tiles = (unsigned)row_tiles, x.first_tile = (unsigned)tiles;
    offset += n_rows * nb;
    tiles += row_tiles * ceil_div(nb, (int64_t)FIT_WARPS);
    HI2_REQUIRE(tiles < ((int64_t)1 << 31), "error_table: too many rows");
  }
  if (row_d != nullptr)
    table_fit_kernel<true><<<(unsigned)tiles, FIT_THREADS, 0, s>>>(w, ldw, d, row_d, n_rows, k, spec, refits, table);
  else
    table_fit_kernel<false><<<(unsigned)tiles, FIT_THREADS, 0, s>>>(w, ldw, d, row_d, n_rows, k, spec, refits, table);
  int rc = check_launch("fit_ladder");
  if (rc != HI2_OK) return rc;
  // the row pass takes as many candidates at a time as their ladders fit in shared memory, six at most
  constexpr int AT_ONCE = 6;
  constexpr int64_t ROOM = ROW_SMEM_MAX / (TABLE_ROW_WARPS * (int64_t)sizeof(TableEntry));
  for (int first = 0; first < n_cand;) {
    int n = 0;
    int64_t entries = 0;
    while (first + n < n_cand && n < AT_ONCE && entries + k / block_host[first + n] <= ROOM)
      entries += k / block_host[first + n], ++n;
    const int smem = (int)(entries * TABLE_ROW_WARPS * (int64_t)sizeof(TableEntry));
    const int64_t want = ceil_div(n_rows, (int64_t)TABLE_ROW_WARPS);
    const unsigned blocks = (unsigned)(want < 148 * 16 ? want : 148 * 16);
    float* en = first == 0 ? energy : nullptr;
#define HI2_TABLE_ROW(NN)                                                                                          \
  case NN:                                                                                                         \
    if (cudaFuncSetAttribute(table_row_kernel<NN>, cudaFuncAttributeMaxDynamicSharedMemorySize, ROW_SMEM_MAX) !=   \
        cudaSuccess)                                                                                               \
      return fail(HI2_ERR_LAUNCH, "quantize_rows: cannot reserve shared memory");                                  \
    table_row_kernel<NN><<<blocks, TABLE_ROW_WARPS * 32, smem, s>>>(w, ldw, d, row_d, n_rows, k, table, first,     \
                                                                    (int)entries, 1.0f, sse, en);                  \
    break
    switch (n) {
      HI2_TABLE_ROW(1);
      HI2_TABLE_ROW(2);
      HI2_TABLE_ROW(3);
      HI2_TABLE_ROW(4);
      HI2_TABLE_ROW(5);
      HI2_TABLE_ROW(6);
    }
#undef HI2_TABLE_ROW
    rc = check_launch("quantize_rows");
    if (rc != HI2_OK) return rc;
    first += n;
  }
  return HI2_OK;
}

extern "C" int hi2_ladder_sse(const uint8_t* codes, const float* w, int64_t ldw, const float* d,
                              const float* lo, const float* st, int64_t ldp, int64_t n_rows,
                              int64_t k, int block, float* sse, void* stream) {
  using namespace hi2;
  HI2_REQUIRE(block_ok(block), "ladder_sse: block must be 16, 32 or 64");
  HI2_REQUIRE(k > 0 && k % block == 0, "ladder_sse: k must be a multiple of the block");
  if (n_rows == 0) return HI2_OK;
  HI2_REQUIRE(codes && w && d && lo && st && sse, "ladder_sse: null pointer");
  HI2_REQUIRE(aligned16(w) && aligned16(d) && ldw % 4 == 0 &&
                  (reinterpret_cast<uintptr_t>(codes) & 3u) == 0,
              "ladder_sse: alignment");
  const unsigned grid = (unsigned)(n_rows < 148 * 16 ? n_rows : 148 * 16);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
#define HI2_SSE(BB) \
  sse_kernel<BB><<<grid, ROW_THREADS, 0, s>>>(codes, w, ldw, d, lo, st, ldp, n_rows, k, sse)
  if (block == 16) HI2_SSE(16);
  if (block == 32) HI2_SSE(32);
  if (block == 64) HI2_SSE(64);
#undef HI2_SSE
  return check_launch("ladder_sse");
}
