// What the two column-sequential block kernels (GPTQ rounding, +-1 refinement) share: up to 128 columns
// of every row are decided one after the other, and each decision changes the row's later columns by
// a multiple of a row of one 128 x 128 block (of the factor U, of Hs).
//
// Four lanes share a row.  The block is taken in windows of 16 columns.  The window's values are kept by
// all four lanes and every lane decides its columns and applies their effect inside the window, so the
// chain from one column to the next carries no exchange between lanes; the columns behind the window
// are dealt out to the lanes in quads (lane h holds columns 16 m + 4 h .. + 3 of every later window)
// and take the window's sixteen effects afterwards, in column order, so every element sees the
// operations of the column-by-column loop in their order.  After a window the quads move down by one
// and every register index stays static.  What a decision needs besides the value is prepared by the
// lane that owns the column, a window ahead, and waits in shared memory; the block is staged there
// once per thread block.  R rows per lane share the reads of the block and give R independent chains.
#pragma once

#include "common.cuh"

namespace hi2 {
namespace row_window {

constexpr int LMAX = 128;
constexpr int WIN = 16;           // columns decided between two updates of the columns behind them
constexpr int QUADS = LMAX / WIN;
constexpr int GROUP_LANES = 4;    // lanes that share a row
constexpr int BLOCK_THREADS = 128;
// Shared memory: the block as windows of 16 rows that start at their own first column, then two floats per
// column, then per row four floats for each of the window's columns and 16 exchange floats (row
// strides of 4 and 20 banks: a 128-bit access of eight rows meets every bank once).
constexpr int U_FLOATS = WIN * QUADS * (LMAX + WIN) / 2;
constexpr int U_DIAG = U_FLOATS;
constexpr int ROW_STAGE = U_DIAG + 2 * LMAX;
constexpr int COLUMN_STRIDE = 4 * WIN + 4, SWAP_STRIDE = WIN + 4;
__host__ __device__ constexpr int window_base(int win) { return WIN * (LMAX * win - (WIN / 2) * win * (win - 1)); }
static_assert(window_base(QUADS) == U_FLOATS, "the windows fill the stage");

template <int R>
constexpr int rows_per_block() {
  return BLOCK_THREADS / GROUP_LANES * R;
}
template <int R>
constexpr int smem_bytes() {
  return (ROW_STAGE + rows_per_block<R>() * (COLUMN_STRIDE + SWAP_STRIDE)) * (int)sizeof(float);
}

// Rows per lane, by how many waves of thread blocks the rows make (four blocks of 32 rows per SM with one
// row per lane, three blocks of 64 with two): a wave of pairs takes 4/3 of the time of a wave of
// single rows.  GPTQ block at K = 2048, one row / two rows per lane: 4096 rows 25 / 42 us, 16384 50 / 52,
// 22016 74 / 64, 32768 89 / 96.
inline bool two_rows_per_lane(int64_t n_rows) {
  int device = 0, sms = 148;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return 3 * ceil_div(n_rows, (int64_t)sms * 4 * 32) > 4 * ceil_div(n_rows, (int64_t)sms * 3 * 64);
}

// (w0, w1) + f * (u0, u1) with the product and the sum rounded separately.  The product is one packed
// multiply; the two additions stay scalar on purpose: a packed multiply feeding a packed add is
// contracted into a packed FMA by the assembler even with contraction switched off, and a fused update
// no longer gives the codes of the reference's separately rounded one.
__device__ __forceinline__ void add_scaled(float& w0, float& w1, float2 f, float u0, float u1) {
  const float2 p = __fmul2_rn(f, make_float2(u0, u1));
  w0 += p.x, w1 += p.y;
}

// The upper triangle (by windows) of the block at `src` into u; complete after cp.async.wait_all and a
// barrier.
__device__ __forceinline__ void stage_block(float* u, const float* src, int64_t ld, int len) {
  for (int idx = threadIdx.x; idx < len * 32; idx += BLOCK_THREADS) {
    const int j = idx >> 5, c = (idx & 31) * 4, win = j / WIN, first = win * WIN;
    if (c < first || c >= len) continue;
    const float* from = src + (int64_t)j * ld + c;
    float* to = u + window_base(win) + (j - first) * (LMAX - first) + (c - first);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from)
                 : "memory");
  }
}

// Column j of the window has its factor f[r]: the later columns of the window add f * row j of the block.
template <int R>
__device__ __forceinline__ void update_window(float (&v)[R][WIN], const float (&f)[R], int j, const float* urow) {
#pragma unroll
  for (int c = 0; c < WIN; c += 4) {
    if (c + 3 <= j) continue;
    const float4 x = *reinterpret_cast<const float4*>(urow + c);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (c > j) {
        const float2 f2 = make_float2(f[r], f[r]);
        add_scaled(v[r][c], v[r][c + 1], f2, x.x, x.y);
        add_scaled(v[r][c + 2], v[r][c + 3], f2, x.z, x.w);
      } else {  // the quad of column j itself
        if (c + 1 > j) v[r][c + 1] = v[r][c + 1] + f[r] * x.y;
        if (c + 2 > j) v[r][c + 2] = v[r][c + 2] + f[r] * x.z;
        v[r][c + 3] = v[r][c + 3] + f[r] * x.w;
      }
    }
  }
}

// The M quads a lane holds behind the window add the window's sixteen effects, in column order; the
// factors (NEGATE: minus them) wait in the exchange floats.
template <int R, int M, bool NEGATE>
__device__ __forceinline__ void update_quads(float4 (&w)[R][QUADS], const float* u, int width, int quad,
                                             const float* const (&swap)[R]) {
#pragma unroll 1
  for (int j = 0; j < WIN; j += 4) {
    float4 e[R];
#pragma unroll
    for (int r = 0; r < R; ++r) e[r] = *reinterpret_cast<const float4*>(swap[r] + j);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float* row = u + (j + t) * width + 4 * quad;
#pragma unroll
      for (int m = 1; m <= M; ++m) {
        const float4 v = *reinterpret_cast<const float4*>(row + WIN * m);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float x = t == 0 ? e[r].x : t == 1 ? e[r].y : t == 2 ? e[r].z : e[r].w;
          const float2 f = NEGATE ? make_float2(-x, -x) : make_float2(x, x);
          add_scaled(w[r][m].x, w[r][m].y, f, v.x, v.y);
          add_scaled(w[r][m].z, w[r][m].w, f, v.z, v.w);
        }
      }
    }
  }
}
// The same for `behind` windows still to come (up to one quad more than there are: it is never used), and
// the move to the next window.
template <int R, bool NEGATE>
__device__ __forceinline__ void update_behind(float4 (&w)[R][QUADS], const float* u, int width, int quad,
                                              const float* const (&swap)[R], int behind) {
  if (behind > 5) update_quads<R, 7, NEGATE>(w, u, width, quad, swap);
  else if (behind > 3) update_quads<R, 5, NEGATE>(w, u, width, quad, swap);
  else if (behind > 1) update_quads<R, 3, NEGATE>(w, u, width, quad, swap);
  else if (behind > 0) update_quads<R, 1, NEGATE>(w, u, width, quad, swap);
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m + 1 < QUADS; ++m) w[r][m] = w[r][m + 1];
}

// hi = tf32(x), lo = tf32(x - hi), round-to-nearest: the operand form of the tensor-core product that
// follows a block (lazy_tc.cu).
__device__ __forceinline__ void tf32_parts(float x, float& hi, float& lo) {
  uint32_t hb, lb;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hb) : "f"(x));
  hi = __uint_as_float(hb);
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lb) : "f"(x - hi));
  lo = __uint_as_float(lb);
}
// Four factors as they are, or (lo given) as their TF32 parts.
__device__ __forceinline__ void store_factors(float* out, float* out_lo, float4 e) {
  if (out_lo == nullptr) {
    *reinterpret_cast<float4*>(out) = e;
    return;
  }
  float4 h, l;
  tf32_parts(e.x, h.x, l.x), tf32_parts(e.y, h.y, l.y), tf32_parts(e.z, h.z, l.z), tf32_parts(e.w, h.w, l.w);
  *reinterpret_cast<float4*>(out) = h;
  *reinterpret_cast<float4*>(out_lo) = l;
}

}  // namespace row_window
}  // namespace hi2
