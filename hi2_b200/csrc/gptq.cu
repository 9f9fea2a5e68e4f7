// Fixed-ladder GPTQ rounding (hi2/gptq_kernel.py:59-127, hi2/hessian.py:267-315).
//
// Block kernel: four lanes per row (see gptq_block_kernel).  Each product, sum and quotient is
// rounded on its own (the library is built without FMA contraction) and wq is rounded to fp16
// before the error is formed, so given the same inputs the codes equal those of the
// column-by-column loop.
//
// Trailing update: wc[:, i2:] -= err1 @ U[i1:i2, i2:], in fp32 FMA arithmetic (gemm.cuh) or as three
// TF32 products (lazy_tc.cu); neighbouring units with one factor share a launch.
#include "gemm.cuh"
#include "row_window.cuh"

#include <vector>

namespace hi2 {

// lazy_tc.cu
int launch_lazy_tc(float* wc, int64_t n_rows, int64_t k, int64_t i1, int64_t col_end, const float* err_hi,
                   const float* err_lo, int64_t lde, const float* u_hi, const float* u_lo, int* status,
                   cudaStream_t stream);
int launch_lazy_group(float* wc, int64_t n_rows, int64_t k, int64_t i1, int blocks, const float* err_hi,
                      const float* err_lo, int64_t lde, const float* u_hi, const float* u_lo, int* status,
                      cudaStream_t stream);

namespace {

using namespace row_window;

// Code and scaled error of one column (hi2/gptq_kernel.py:88-101) with true divisions.
__device__ __noinline__ float2 round_careful(float col, float lo, float st, float ud, float nm) {
  const float safe = (st == 0.0f) ? 1.0f : st;
  float q = rintf(__fdiv_rn(col - lo, safe));
  q = (q < 0.0f) ? 0.0f : q;
  q = (q > nm) ? nm : q;
  if (st == 0.0f) q = 0.0f;
  const float wq = round_f16(lo + q * st);
  return make_float2(q, __fdiv_rn(col - wq, ud));
}

// The same from prepared values: ladder = (lo, st, 1 / st, highest code: 0 for st == 0), diag = (U_jj,
// 1 / U_jj).  a * (1 / st) is within 3 ulp of the quotient and rounds to the same integer unless it lies
// within a few ulp of a half-integer (below 256, where every ladder ends, those are less than 1e-4);
// such columns, NaNs, and ladders and pivots whose reciprocal is not usable (stored as NaN) take the
// careful path.  The integer is taken by adding and removing 1.5 * 2^23, which rounds to nearest even
// below 2^22 and keeps anything larger beyond every ladder.  The error's quotient is finished with
// Markstein's fused correction and is the IEEE one.
__device__ __forceinline__ void round_column(float col, float4 ladder, float2 diag, float nm, float& q_out,
                                             float& e_out) {
  const float t = (col - ladder.x) * ladder.z;
  float q = (t + 12582912.0f) - 12582912.0f;
  const bool clear = fabsf(fabsf(t - q) - 0.5f) >= 2.5e-4f;  // false for NaN
  q = fminf(fmaxf(q, 0.0f), ladder.w);
  const float num = col - round_f16(ladder.x + q * ladder.y);
  const float q0 = num * diag.y;
  q_out = q;
  e_out = fmaf(fmaf(-q0, diag.x, num), diag.y, q0);
  if (!clear) {
    const float2 r = round_careful(col, ladder.x, ladder.y, diag.x, nm);
    q_out = r.x, e_out = r.y;
  }
}

// One lazy block: up to 128 columns of every row, rounded column by column, in the mapping of
// row_window.cuh.  The prepared values of a column are its ladder and the ladder's reciprocal.
// What bounds it: few rows, the chain (about 110 cycles a column); many rows, shared-memory reads of the
// factor.  One lane per row with the 128 columns in its registers was bound by the chain at every size
// and left most SMs idle at a few thousand rows; a block, lane per row -> this: 256 rows 79 -> 23 us,
// 4096 81 -> 23, 11008 88 -> 39, 22016 107 -> 62, 32768 163 -> 88.
// Rows of one thread block that read different factors (a block that straddles two tensors) are
// served one factor after the other: everybody computes, only the rows of that factor store.
template <int R, bool WITH_COMP, bool SPLIT>
__global__ void __launch_bounds__(BLOCK_THREADS, (R == 1 ? 4 : 3))
gptq_block_kernel(const float* __restrict__ wc, int64_t n_rows, int64_t k, int64_t i1, int len,
                  float* __restrict__ err, float* __restrict__ err_lo, int64_t lde, uint8_t* __restrict__ codes,
                  const float* __restrict__ lo, const float* __restrict__ st, int64_t ldp,
                  const int32_t* __restrict__ row_grp, const int64_t* __restrict__ u_ptrs,
                  const int32_t* __restrict__ blk, const float* __restrict__ nmax,
                  float* __restrict__ comp) {
  extern __shared__ __align__(16) float gptq_smem[];
  __shared__ unsigned long long next_factor;
  const int lane = threadIdx.x & 31, quad = lane & 3;
  const int row0 = (threadIdx.x >> 5) * 8 * R + (lane >> 2);  // this lane's rows of the block: row0 + 8 r
  float* u = gptq_smem;
  const float2* diag = reinterpret_cast<const float2*>(gptq_smem + U_DIAG);
  float* ladders = gptq_smem + ROW_STAGE;
  float* swaps = ladders + rows_per_block<R>() * COLUMN_STRIDE;
  const int windows = len / WIN;

  int64_t row[R];
  bool live[R], done[R];
  unsigned long long factor_of[R];
  float nm[R];
  int group[R];
  const float* swap[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t raw = (int64_t)blockIdx.x * rows_per_block<R>() + row0 + 8 * r;
    live[r] = raw < n_rows;
    row[r] = live[r] ? raw : n_rows - 1;  // spare lanes shadow the last row and store nothing
    group[r] = row_grp[row[r]];
    factor_of[r] = (unsigned long long)u_ptrs[group[r]];
    nm[r] = nmax[group[r]];
    done[r] = false;
    swap[r] = swaps + (row0 + 8 * r) * SWAP_STRIDE;
  }

  while (true) {
    if (threadIdx.x == 0) next_factor = ~0ull;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (!done[r]) atomicMin(&next_factor, factor_of[r]);
    __syncthreads();
    const unsigned long long factor = next_factor;
    if (factor == ~0ull) break;
    {
      const float* src = reinterpret_cast<const float*>(factor) + i1 * k + i1;
      stage_block(u, src, k, len);
      for (int j = threadIdx.x; j < len; j += BLOCK_THREADS) {
        const float ud = src[(int64_t)j * k + j];
        const Recip rc = make_recip(ud);
        reinterpret_cast<float2*>(gptq_smem + U_DIAG)[j] = make_float2(ud, rc.fast ? rc.r : __int_as_float(0x7fc00000));
      }
    }
    float4 w[R][QUADS];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int m = 0; m < QUADS; ++m)
        w[r][m] = WIN * m < len ? *reinterpret_cast<const float4*>(wc + row[r] * k + i1 + WIN * m + 4 * quad)
                                : make_float4(0.f, 0.f, 0.f, 0.f);
    // ladders of this lane's quad of window 0, and the block indices of window 1 behind them
    float lo_n[R][4], st_n[R][4];
    int4 blk_n[R] = {};
    auto fetch_ladders = [&](int r) {
      const float *l = lo + row[r] * ldp, *s = st + row[r] * ldp;
      lo_n[r][0] = l[blk_n[r].x], lo_n[r][1] = l[blk_n[r].y], lo_n[r][2] = l[blk_n[r].z], lo_n[r][3] = l[blk_n[r].w];
      st_n[r][0] = s[blk_n[r].x], st_n[r][1] = s[blk_n[r].y], st_n[r][2] = s[blk_n[r].z], st_n[r][3] = s[blk_n[r].w];
    };
    auto fetch_blocks = [&](int r, int win) {
      blk_n[r] = *reinterpret_cast<const int4*>(blk + (int64_t)group[r] * k + i1 + WIN * min(win, windows - 1) + 4 * quad);
    };
#pragma unroll
    for (int r = 0; r < R; ++r) {
      fetch_blocks(r, 0);
      fetch_ladders(r);
      fetch_blocks(r, 1);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

#pragma unroll 1
    for (int win = 0; win < windows; ++win) {
      // ---- the window's values and ladders for all four lanes
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float* lad = ladders + (row0 + 8 * r) * COLUMN_STRIDE + 16 * quad;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float s = st_n[r][t];
          const float safe = s == 0.0f ? 1.0f : s, pivot = diag[WIN * win + 4 * quad + t].y;
          float z;  // within an ulp of 1 / safe, which round_column's margin covers
          asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(z) : "f"(safe));
          if (!(fabsf(safe) > 1e-18f && fabsf(safe) < 1e18f && pivot == pivot)) z = __int_as_float(0x7fc00000);
          *reinterpret_cast<float4*>(lad + 4 * t) = make_float4(lo_n[r][t], s, z, s == 0.0f ? 0.0f : nm[r]);
        }
        *reinterpret_cast<float4*>(const_cast<float*>(swap[r]) + 4 * quad) = w[r][0];
      }
      __syncwarp();
      float v[R][WIN];
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int t = 0; t < WIN; t += 4) {
          const float4 x = *reinterpret_cast<const float4*>(swap[r] + t);
          v[r][t] = x.x, v[r][t + 1] = x.y, v[r][t + 2] = x.z, v[r][t + 3] = x.w;
        }
        if (win + 1 < windows) {  // loads for the next window, in flight during this one
          fetch_ladders(r);
          fetch_blocks(r, win + 2);
        }
      }
      __syncwarp();  // the exchange floats take the errors from here on
      const int width = LMAX - WIN * win;
      const float* uw = u + window_base(win);
      uint32_t code[R][4];
      float seen[WITH_COMP ? R : 1][WITH_COMP ? WIN : 1];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float e[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r) code[r][q] = 0;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int j = 4 * q + t;
          const float2 dj = diag[WIN * win + j];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float4 lad = *reinterpret_cast<const float4*>(ladders + (row0 + 8 * r) * COLUMN_STRIDE + 4 * j);
            float code_j;
            if (WITH_COMP) seen[r][j] = v[r][j];
            round_column(v[r][j], lad, dj, nm[r], code_j, e[r][t]);
            code[r][q] |= (uint32_t)code_j << (8 * t);
          }
          float f[R];
#pragma unroll
          for (int r = 0; r < R; ++r) f[r] = -e[r][t];
          update_window<R>(v, f, j, uw + j * width);
        }
        if (quad == 0) {
#pragma unroll
          for (int r = 0; r < R; ++r)
            *reinterpret_cast<float4*>(const_cast<float*>(swap[r]) + 4 * q) = make_float4(e[r][0], e[r][1], e[r][2], e[r][3]);
        }
      }
      __syncwarp();
      // ---- outputs: each lane stores its quad of the window
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (!live[r] || done[r] || factor_of[r] != factor) continue;
        const int64_t at = WIN * win + 4 * quad;
        const float4 e = *reinterpret_cast<const float4*>(swap[r] + 4 * quad);
        store_factors(err + row[r] * lde + at, SPLIT ? err_lo + row[r] * lde + at : nullptr, e);
        const uint32_t c01 = quad & 1 ? code[r][1] : code[r][0], c23 = quad & 1 ? code[r][3] : code[r][2];
        *reinterpret_cast<uint32_t*>(codes + row[r] * k + i1 + at) = quad & 2 ? c23 : c01;
        if (WITH_COMP) {
          float x[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float x01 = quad & 1 ? seen[r][4 + t] : seen[r][t], x23 = quad & 1 ? seen[r][12 + t] : seen[r][8 + t];
            x[t] = quad & 2 ? x23 : x01;
          }
          *reinterpret_cast<float4*>(comp + row[r] * k + i1 + at) = make_float4(x[0], x[1], x[2], x[3]);
        }
      }
      update_behind<R, true>(w, uw, width, quad, swap, windows - 1 - win);
      __syncwarp();  // the exchange floats are overwritten next
    }
#pragma unroll
    for (int r = 0; r < R; ++r) done[r] = done[r] || factor_of[r] == factor;
    __syncthreads();  // the staged block is replaced in the next round
  }
}

template <int R, bool WITH_COMP, bool SPLIT>
int launch_block_as(const float* wc, int64_t n_rows, int64_t k, int64_t i1, int len, float* err, float* err_lo,
                    int64_t lde, uint8_t* codes, const float* lo, const float* st, int64_t ldp, const int32_t* row_grp,
                    const int64_t* u_ptrs, const int32_t* blk, const float* nmax, float* comp, cudaStream_t stream) {
  constexpr int rows = rows_per_block<R>(), smem = smem_bytes<R>();
  auto kernel = gptq_block_kernel<R, WITH_COMP, SPLIT>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return fail(HI2_ERR_LAUNCH, "gptq_block: cannot reserve shared memory");
  // Not a launch_link: set up while an update still holds most SMs, the thread blocks would pile up on the
  // few that are free (column loop of 4096 x 4096 1.7 -> 2.3 ms).
  kernel<<<(unsigned)ceil_div(n_rows, (int64_t)rows), BLOCK_THREADS, smem, stream>>>(
      wc, n_rows, k, i1, len, err, err_lo, lde, codes, lo, st, ldp, row_grp, u_ptrs, blk, nmax, comp);
  return check_launch("gptq_block");
}

// err_lo null: err (leading dimension lde) receives the errors; else err and err_lo their TF32 parts.
int launch_block(const float* wc, int64_t n_rows, int64_t k, int64_t i1, int len, float* err, float* err_lo,
                 int64_t lde, uint8_t* codes, const float* lo, const float* st, int64_t ldp,
                 const int32_t* row_grp, const int64_t* u_ptrs, const int32_t* blk,
                 const float* nmax, float* comp, cudaStream_t stream) {
#define HI2_GPTQ_BLOCK(RR, CC, SS)                                                                              \
  return launch_block_as<RR, CC, SS>(wc, n_rows, k, i1, len, err, err_lo, lde, codes, lo, st, ldp, row_grp, u_ptrs, blk, \
                                     nmax, comp, stream)
  const bool pair = two_rows_per_lane(n_rows);
  if (comp != nullptr) {
    if (err_lo != nullptr) {
      if (pair) HI2_GPTQ_BLOCK(2, true, true);
      HI2_GPTQ_BLOCK(1, true, true);
    }
    if (pair) HI2_GPTQ_BLOCK(2, true, false);
    HI2_GPTQ_BLOCK(1, true, false);
  }
  if (err_lo != nullptr) {
    if (pair) HI2_GPTQ_BLOCK(2, false, true);
    HI2_GPTQ_BLOCK(1, false, true);
  }
  if (pair) HI2_GPTQ_BLOCK(2, false, false);
  HI2_GPTQ_BLOCK(1, false, false);
#undef HI2_GPTQ_BLOCK
}

// Consecutive rows with one factor: units of one tensor (its candidate groups), and of tensors that
// read the same input, lie next to each other, and their trailing updates are one product.
struct Span {
  int64_t r0, r1, factor;
};
std::vector<Span> factor_spans(int n_units, const int64_t* unit_rows, const int64_t* unit_factor) {
  std::vector<Span> spans;
  for (int un = 0; un < n_units; ++un) {
    const int64_t r0 = unit_rows[un], r1 = unit_rows[un + 1];
    if (r1 <= r0) continue;
    if (!spans.empty() && spans.back().factor == unit_factor[un] && spans.back().r1 == r0) spans.back().r1 = r1;
    else spans.push_back({r0, r1, unit_factor[un]});
  }
  return spans;
}

int launch_lazy(float* wc, int64_t n_rows, int64_t k, int64_t i1, int64_t i2, const float* err1,
                const float* u, cudaStream_t stream) {
  GemmArgs<float, float, float> p;
  p.m = n_rows, p.n = k - i2, p.kk = i2 - i1;
  p.alpha = -1.0f, p.beta = 1.0f;
  p.a = err1, p.lda = i2 - i1;
  p.b = u + i1 * k + i2, p.ldb = k;
  p.c = wc + i2, p.ldc = k;
  p.flags = 0;
  return launch_gemm_async<float, 8, 8, 16>(false, false, p, stream, "gptq_lazy_update");
}

int check_block_args(const float* wc, int64_t n_rows, int64_t k, int64_t i1, int len,
                     const float* err1, const uint8_t* codes, const float* lo, const float* st,
                     int64_t ldp, const int32_t* row_grp, const int64_t* u_ptrs, const int32_t* blk,
                     const float* nmax, const float* comp) {
  HI2_REQUIRE(k > 0 && k % 16 == 0, "gptq_block: k must be a positive multiple of 16");
  HI2_REQUIRE(len > 0 && len <= LMAX && len % 16 == 0, "gptq_block: block length must be 16..128");
  HI2_REQUIRE(i1 >= 0 && i1 % 16 == 0 && i1 + len <= k, "gptq_block: block outside the row");
  HI2_REQUIRE(wc && err1 && codes && lo && st && row_grp && u_ptrs && blk && nmax,
              "gptq_block: null pointer");
  HI2_REQUIRE(aligned16(wc) && aligned16(err1) && aligned16(blk) && (comp == nullptr || aligned16(comp)),
              "gptq_block: wc, err1, blk and comp must be 16-byte aligned");
  HI2_REQUIRE((reinterpret_cast<uintptr_t>(codes) & 3u) == 0, "gptq_block: codes must be 4-byte aligned");
  HI2_REQUIRE(ldp > 0, "gptq_block: ldp");
  (void)n_rows;
  return HI2_OK;
}

}  // namespace
}  // namespace hi2

extern "C" int hi2_gptq_block(const float* wc, int64_t n_rows, int64_t k, int64_t i1, int len,
                              float* err1, uint8_t* codes, const float* lo, const float* st,
                              int64_t ldp, const int32_t* row_grp, const int64_t* u_ptrs,
                              const int32_t* blk, const float* nmax, float* comp, void* stream) {
  using namespace hi2;
  if (n_rows == 0) return HI2_OK;
  int rc = check_block_args(wc, n_rows, k, i1, len, err1, codes, lo, st, ldp, row_grp, u_ptrs, blk,
                            nmax, comp);
  if (rc != HI2_OK) return rc;
  return launch_block(wc, n_rows, k, i1, len, err1, nullptr, len, codes, lo, st, ldp, row_grp, u_ptrs, blk, nmax,
                      comp, static_cast<cudaStream_t>(stream));
}

extern "C" int hi2_gptq_lazy_update(float* wc, int64_t n_rows, int64_t k, int64_t i1, int64_t i2,
                                    const float* err1, const float* u, void* stream) {
  using namespace hi2;
  HI2_REQUIRE(k > 0 && 0 <= i1 && i1 < i2 && i2 <= k, "gptq_lazy_update: bad block range");
  if (n_rows == 0 || i2 == k) return HI2_OK;
  HI2_REQUIRE(wc && err1 && u, "gptq_lazy_update: null pointer");
  return launch_lazy(wc, n_rows, k, i1, i2, err1, u, static_cast<cudaStream_t>(stream));
}

extern "C" int hi2_gptq_round(float* wc, int64_t n_rows, int64_t k, float* err1, uint8_t* codes,
                              const float* lo, const float* st, int64_t ldp,
                              const int32_t* row_grp, const int64_t* u_ptrs, const int32_t* blk,
                              const float* nmax, float* comp, int n_units,
                              const int64_t* unit_rows_host, const int64_t* u_host, void* stream) {
  using namespace hi2;
  if (n_rows == 0) return HI2_OK;
  HI2_REQUIRE(n_units >= 1 && unit_rows_host && u_host, "gptq_round: unit table missing");
  HI2_REQUIRE(unit_rows_host[0] == 0 && unit_rows_host[n_units] == n_rows,
              "gptq_round: units must cover the rows");
  for (int un = 0; un < n_units; ++un)  // the blocks are staged with 128-bit copies
    HI2_REQUIRE(aligned16(reinterpret_cast<const void*>(u_host[un])), "gptq_round: factors must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const std::vector<Span> spans = factor_spans(n_units, unit_rows_host, u_host);
  ChainGraph chain(s, ceil_div(k, LMAX) * (1 + (int64_t)spans.size()));  // the segments and their trailing updates
  auto enqueue = [&]() -> int {
    for (int64_t i1 = 0; i1 < k; i1 += LMAX) {
      const int64_t i2 = (i1 + LMAX < k) ? i1 + LMAX : k;
      const int len = (int)(i2 - i1);
      int rc = check_block_args(wc, n_rows, k, i1, len, err1, codes, lo, st, ldp, row_grp, u_ptrs,
                                blk, nmax, comp);
      if (rc != HI2_OK) return rc;
      rc = launch_block(wc, n_rows, k, i1, len, err1, nullptr, len, codes, lo, st, ldp, row_grp, u_ptrs, blk, nmax,
                        comp, s);
      if (rc != HI2_OK) return rc;
      if (i2 == k) break;
      for (const Span& x : spans) {
        rc = launch_lazy(wc + x.r0 * k, x.r1 - x.r0, k, i1, i2, err1 + x.r0 * len,
                         reinterpret_cast<const float*>(x.factor), s);
        if (rc != HI2_OK) return rc;
      }
    }
    return HI2_OK;
  };
  return chain.finish(enqueue(), "gptq_round");
}

extern "C" int hi2_gptq_lazy_update_tc(float* wc, int64_t n_rows, int64_t k, int64_t i1,
                                       const float* err_split, const float* u_split, int32_t* status,
                                       void* stream) {
  using namespace hi2;
  HI2_REQUIRE(k > 0 && k % 4 == 0 && i1 >= 0 && i1 % 4 == 0 && i1 + LMAX <= k,
              "gptq_lazy_update_tc: bad block range");
  if (n_rows == 0 || i1 + LMAX == k) return HI2_OK;
  HI2_REQUIRE(wc && err_split && u_split && status, "gptq_lazy_update_tc: null pointer");
  HI2_REQUIRE(aligned16(wc) && aligned16(err_split) && aligned16(u_split), "gptq_lazy_update_tc: alignment");
  return launch_lazy_tc(wc, n_rows, k, i1, k, err_split, err_split + n_rows * LMAX, LMAX, u_split, u_split + k * k,
                        reinterpret_cast<int*>(status), static_cast<cudaStream_t>(stream));
}

extern "C" int hi2_gptq_round_tc_grouped(float* wc, int64_t n_rows, int64_t k, float* err_split, int64_t err_columns,
                                         uint8_t* codes, const float* lo, const float* st, int64_t ldp,
                                         const int32_t* row_grp, const int64_t* u_ptrs, const int32_t* blk,
                                         const float* nmax, float* comp, int n_units,
                                         const int64_t* unit_rows_host, const int64_t* u_split_host,
                                         int32_t* status, void* stream) {
  using namespace hi2;
  if (n_rows == 0) return HI2_OK;
  HI2_REQUIRE(n_units >= 1 && unit_rows_host && u_split_host, "gptq_round_tc: unit table missing");
  HI2_REQUIRE(unit_rows_host[0] == 0 && unit_rows_host[n_units] == n_rows,
              "gptq_round_tc: units must cover the rows");
  HI2_REQUIRE(err_split && status && aligned16(err_split), "gptq_round_tc: scratch missing or unaligned");
  HI2_REQUIRE(k % 4 == 0, "gptq_round_tc: k must be a multiple of 4");
  HI2_REQUIRE(err_columns >= LMAX && err_columns % LMAX == 0, "gptq_round_tc: err_columns must be a multiple of 128");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  float* err_hi = err_split;
  float* err_lo = err_split + n_rows * err_columns;
  int* word = reinterpret_cast<int*>(status);
  const std::vector<Span> spans = factor_spans(n_units, unit_rows_host, u_split_host);
  ChainGraph chain(s, ceil_div(k, LMAX) * (1 + (int64_t)spans.size()));  // the segments and their trailing updates
  auto enqueue = [&]() -> int {
    if (cudaMemsetAsync(status, 0, sizeof(int32_t), s) != cudaSuccess)
      return fail(HI2_ERR_LAUNCH, "gptq_round_tc: memset failed");
    for (int64_t g0 = 0; g0 < k; g0 += err_columns) {
      const int64_t g1 = (g0 + err_columns < k) ? g0 + err_columns : k;
      for (int64_t i1 = g0; i1 < g1; i1 += LMAX) {
        const int64_t i2 = (i1 + LMAX < k) ? i1 + LMAX : k;
        const int len = (int)(i2 - i1);
        float *eh = err_hi + (i1 - g0), *el = err_lo + (i1 - g0);
        int rc = check_block_args(wc, n_rows, k, i1, len, eh, codes, lo, st, ldp, row_grp, u_ptrs, blk, nmax, comp);
        if (rc != HI2_OK) return rc;
        // the block leaves its errors as the TF32 parts the trailing updates take
        rc = launch_block(wc, n_rows, k, i1, len, eh, el, err_columns, codes, lo, st, ldp, row_grp, u_ptrs, blk, nmax,
                          comp, s);
        if (rc != HI2_OK) return rc;
        if (i2 >= g1) break;  // a block shorter than 128 columns is always the last one
        for (const Span& x : spans) {  // the rest of the group needs this block's errors now
          const float* u_hi = reinterpret_cast<const float*>(x.factor);
          rc = launch_lazy_tc(wc + x.r0 * k, x.r1 - x.r0, k, i1, g1, eh + x.r0 * err_columns, el + x.r0 * err_columns,
                              err_columns, u_hi, u_hi + k * k, word, s);
          if (rc != HI2_OK) return rc;
        }
      }
      if (g1 == k) break;
      for (const Span& x : spans) {  // the columns behind it take all of its blocks in one pass
        const float* u_hi = reinterpret_cast<const float*>(x.factor);
        const float *eh = err_hi + x.r0 * err_columns, *el = err_lo + x.r0 * err_columns;
        const int blocks = (int)(err_columns / LMAX);
        int rc = blocks == 1 ? launch_lazy_tc(wc + x.r0 * k, x.r1 - x.r0, k, g0, k, eh, el, err_columns, u_hi,
                                              u_hi + k * k, word, s)
                             : launch_lazy_group(wc + x.r0 * k, x.r1 - x.r0, k, g0, blocks, eh, el, err_columns, u_hi,
                                                 u_hi + k * k, word, s);
        if (rc != HI2_OK) return rc;
      }
    }
    return HI2_OK;
  };
  return chain.finish(enqueue(), "gptq_round_tc");
}

extern "C" int hi2_gptq_round_tc(float* wc, int64_t n_rows, int64_t k, float* err1, float* err_split,
                                 uint8_t* codes, const float* lo, const float* st, int64_t ldp,
                                 const int32_t* row_grp, const int64_t* u_ptrs, const int32_t* blk,
                                 const float* nmax, float* comp, int n_units,
                                 const int64_t* unit_rows_host, const int64_t* u_split_host,
                                 int32_t* status, void* stream) {
  (void)err1;
  return hi2_gptq_round_tc_grouped(wc, n_rows, k, err_split, hi2::row_window::LMAX, codes, lo, st, ldp, row_grp, u_ptrs, blk, nmax,
                                   comp, n_units, unit_rows_host, u_split_host, status, stream);
}

extern "C" int hi2_gemm_f32(int trans_a, int trans_b, int64_t m, int64_t n, int64_t kk, float alpha,
                            const float* a, int64_t lda, const float* b, int64_t ldb, float beta,
                            float* c, int64_t ldc, void* stream) {
  using namespace hi2;
  HI2_REQUIRE(m >= 0 && n >= 0 && kk >= 0, "gemm_f32: negative size");
  if (m == 0 || n == 0) return HI2_OK;
  HI2_REQUIRE(c && (kk == 0 || (a && b)), "gemm_f32: null pointer");
  GemmArgs<float, float, float> p;
  p.m = m, p.n = n, p.kk = kk, p.alpha = alpha, p.beta = beta;
  p.a = a, p.lda = lda, p.b = b, p.ldb = ldb, p.c = c, p.ldc = ldc, p.flags = 0;
  return launch_gemm_async<float, 8, 8, 16>(trans_a != 0, trans_b != 0, p,
                                            static_cast<cudaStream_t>(stream), "gemm_f32");
}
