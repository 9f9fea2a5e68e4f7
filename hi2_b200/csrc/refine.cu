// One block of columns of the +-1 refinement sweep (hi2/refine_kernel.py:51-120).
//
// The mapping is that of row_window.cuh: four lanes per row, windows of 16 columns.  A column's move is
// decided exactly as the reference kernel decides it: gain = -((2*dw)*g + (dw*dw)*H_jj), each operation
// rounded on its own; ties go to +1; NaN never moves; a move adds dw * Hs[j, q] (product and sum
// rounded separately) to every later column q of the block, in column order.  A column that does not
// move adds dw = 0, which leaves g as it is.  2 dw and (dw dw) H_jj of both moves do not depend on g and
// are prepared a window ahead, so the chain of a column is two products, two sums and two comparisons.
// Measured per block of 4096 x 128, us: a warp per row with a shuffle per column 47, this 19.
#include "gemm.cuh"
#include "row_window.cuh"

namespace hi2 {
// lazy_tc.cu; flag 32: the product is added to c
int launch_gemm_tc2(int64_t m, int64_t n, int64_t kk, const float* a_hi, const float* a_lo, int64_t lda,
                    const float* b_hi, const float* b_lo, int64_t ldb, float* c, int64_t ldc, int flags,
                    int* status, cudaStream_t stream);
namespace {

using namespace row_window;
constexpr int GT_ADD = 32;

template <int R>
__global__ void __launch_bounds__(BLOCK_THREADS, (R == 1 ? 4 : 3))
refine_block_kernel(const float* __restrict__ gb, int64_t ldg, int len, float* __restrict__ c,
                    const float* __restrict__ lo, const float* __restrict__ st,
                    const float* __restrict__ top, const float* __restrict__ hs, int64_t n_rows,
                    int64_t k, int64_t b0, float* __restrict__ dwb, float* __restrict__ dw_lo, int64_t lddw,
                    int32_t* __restrict__ moved_any) {
  extern __shared__ __align__(16) float refine_smem[];
  const int lane = threadIdx.x & 31, quad = lane & 3;
  const int row0 = (threadIdx.x >> 5) * 8 * R + (lane >> 2);  // this lane's rows of the block: row0 + 8 r
  float* u = refine_smem;
  float* columns = refine_smem + ROW_STAGE;
  float* swaps = columns + rows_per_block<R>() * COLUMN_STRIDE;
  const int windows = len / WIN;
  stage_block(u, hs + b0 * k + b0, k, len);

  int64_t row[R];
  bool live[R];
  float tp[R];
  const float* swap[R];
  float4 w[R][QUADS], code[R], lo_n[R], st_n[R];  // code, lo, st: of this lane's quad of the next window
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t raw = (int64_t)blockIdx.x * rows_per_block<R>() + row0 + 8 * r;
    live[r] = raw < n_rows;
    row[r] = live[r] ? raw : n_rows - 1;  // spare lanes shadow the last row and store nothing
    tp[r] = top[row[r]];
    swap[r] = swaps + (row0 + 8 * r) * SWAP_STRIDE;
#pragma unroll
    for (int m = 0; m < QUADS; ++m)
      w[r][m] = WIN * m < len ? *reinterpret_cast<const float4*>(gb + row[r] * ldg + WIN * m + 4 * quad)
                              : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  auto fetch = [&](int r, int win) {
    const int64_t at = row[r] * k + b0 + WIN * win + 4 * quad;
    code[r] = *reinterpret_cast<const float4*>(c + at);
    lo_n[r] = *reinterpret_cast<const float4*>(lo + at);
    st_n[r] = *reinterpret_cast<const float4*>(st + at);
  };
#pragma unroll
  for (int r = 0; r < R; ++r) fetch(r, 0);
  bool any = false;  // a live row of this lane has moved
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

#pragma unroll 1
  for (int win = 0; win < windows; ++win) {
    const int width = LMAX - WIN * win;
    const float* uw = u + window_base(win);
    float4 now_code[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float cs[4] = {code[r].x, code[r].y, code[r].z, code[r].w}, ls[4] = {lo_n[r].x, lo_n[r].y, lo_n[r].z, lo_n[r].w},
                  ss[4] = {st_n[r].x, st_n[r].y, st_n[r].z, st_n[r].w};
      float* col = columns + (row0 + 8 * r) * COLUMN_STRIDE + 16 * quad;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float hd = uw[(4 * quad + t) * width + 4 * quad + t];
        const float now = round_f16(ls[t] + cs[t] * ss[t]);
        const float cp = cs[t] + 1.0f, cm = cs[t] - 1.0f;
        const bool okp = (cp >= 0.0f) && (cp <= tp[r]) && (ss[t] > 0.0f);
        const bool okm = (cm >= 0.0f) && (cm <= tp[r]) && (ss[t] > 0.0f);
        const float dwp = round_f16(ls[t] + cp * ss[t]) - now, dwm = round_f16(ls[t] + cm * ss[t]) - now;
        // an infinite second term marks a move that is not open
        *reinterpret_cast<float4*>(col + 4 * t) = make_float4(2.0f * dwp, okp ? (dwp * dwp) * hd : INFINITY, 2.0f * dwm,
                                                              okm ? (dwm * dwm) * hd : INFINITY);
      }
      *reinterpret_cast<float4*>(const_cast<float*>(swap[r]) + 4 * quad) = w[r][0];
      now_code[r] = code[r];
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
      if (win + 1 < windows) fetch(r, win + 1);  // in flight during this window
    }
    __syncwarp();  // the exchange floats take the changes from here on
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float dw[R][4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int j = 4 * q + t;
        float f[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float4 m = *reinterpret_cast<const float4*>(columns + (row0 + 8 * r) * COLUMN_STRIDE + 4 * j);
          const float gp = m.y == INFINITY ? -INFINITY : -(m.x * v[r][j] + m.y);
          const float gm = m.w == INFINITY ? -INFINITY : -(m.z * v[r][j] + m.w);
          const bool minus = gm > gp;
          f[r] = (minus ? gm : gp) > 0.0f ? 0.5f * (minus ? m.z : m.x) : 0.0f;
          dw[r][t] = f[r];
        }
        update_window<R>(v, f, j, uw + j * width);
      }
      if (quad == 0) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          *reinterpret_cast<float4*>(const_cast<float*>(swap[r]) + 4 * q) = make_float4(dw[r][0], dw[r][1], dw[r][2], dw[r][3]);
      }
    }
    __syncwarp();
    // each lane stores its quad; a move up has dw > 0, a move down dw < 0, and a move of 0 gains nothing
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!live[r]) continue;
      const int at = WIN * win + 4 * quad;
      const float4 d = *reinterpret_cast<const float4*>(swap[r] + 4 * quad);
      any = any || d.x != 0.0f || d.y != 0.0f || d.z != 0.0f || d.w != 0.0f;
      auto moved = [](float code_j, float dw_j) { return dw_j > 0.0f ? code_j + 1.0f : (dw_j < 0.0f ? code_j - 1.0f : code_j); };
      *reinterpret_cast<float4*>(c + row[r] * k + b0 + at) =
          make_float4(moved(now_code[r].x, d.x), moved(now_code[r].y, d.y), moved(now_code[r].z, d.z), moved(now_code[r].w, d.w));
      store_factors(dwb + row[r] * lddw + at, dw_lo ? dw_lo + row[r] * lddw + at : nullptr, d);
    }
    update_behind<R, false>(w, uw, width, quad, swap, windows - 1 - win);
    __syncwarp();  // the exchange floats are overwritten next
  }
  if (moved_any != nullptr && any) *moved_any = 1;
}

// What the sweeps start from, for one group of rows in one pass: codes as fp32, the ladder of every column
// (decoded as hi2/format.py:45-60: lo = fp16(fma(byte, lo_scale, lo_min)), step = fp16(byte * step_scale)),
// and the error e = fp16(lo + c step) - w, as it is or as its TF32 parts.  Bound by memory: 20 bytes
// written (16 without the low part) and 5 read per weight; a dozen elementwise passes before, 650 -> 67
// us for 4096 x 4096.
__global__ void __launch_bounds__(256)
refine_prepare_kernel(const float* __restrict__ w, int64_t ldw, const uint8_t* __restrict__ codes,
                      const uint8_t* __restrict__ params, const uint16_t* __restrict__ consts, int shift, int64_t n_rows,
                      int64_t k, float* __restrict__ c, float* __restrict__ lo_x, float* __restrict__ st_x,
                      float* __restrict__ e, float* __restrict__ e_lo) {
  const int64_t j = ((int64_t)blockIdx.y * 256 + threadIdx.x) * 4;
  if (j >= k) return;
  for (int64_t row = blockIdx.x; row < n_rows; row += gridDim.x) {
    const float lm = __half2float(__ushort_as_half(consts[row * 3])), ls = __half2float(__ushort_as_half(consts[row * 3 + 1])),
                ss = __half2float(__ushort_as_half(consts[row * 3 + 2]));
    const uchar2 p = *reinterpret_cast<const uchar2*>(params + (row * (k >> shift) + (j >> shift)) * 2);
    const float lo = round_f16(fmaf((float)p.x, ls, lm)), st = round_f16((float)p.y * ss);
    const uchar4 q = *reinterpret_cast<const uchar4*>(codes + row * k + j);
    const float4 v = *reinterpret_cast<const float4*>(w + row * ldw + j);
    const float4 cf = make_float4((float)q.x, (float)q.y, (float)q.z, (float)q.w);
    const int64_t at = row * k + j;
    *reinterpret_cast<float4*>(c + at) = cf;
    *reinterpret_cast<float4*>(lo_x + at) = make_float4(lo, lo, lo, lo);
    *reinterpret_cast<float4*>(st_x + at) = make_float4(st, st, st, st);
    store_factors(e + at, e_lo ? e_lo + at : nullptr,
                  make_float4(round_f16(lo + cf.x * st) - v.x, round_f16(lo + cf.y * st) - v.y,
                              round_f16(lo + cf.z * st) - v.z, round_f16(lo + cf.w * st) - v.w));
  }
}

template <int R>
int launch_refine_as(const float* gb, int64_t ldg, int len, float* c, const float* lo, const float* st,
                     const float* top, const float* hs, int64_t n_rows, int64_t k, int64_t b0, float* dwb,
                     float* dw_lo, int64_t lddw, int32_t* moved, cudaStream_t stream) {
  if (cudaFuncSetAttribute(refine_block_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<R>()) !=
      cudaSuccess)
    return fail(HI2_ERR_LAUNCH, "refine_block: cannot reserve shared memory");
  refine_block_kernel<R><<<(unsigned)ceil_div(n_rows, (int64_t)rows_per_block<R>()), BLOCK_THREADS, smem_bytes<R>(), stream>>>(
      gb, ldg, len, c, lo, st, top, hs, n_rows, k, b0, dwb, dw_lo, lddw, moved);
  return check_launch("refine_block");
}
int launch_refine_block(const float* gb, int64_t ldg, int len, float* c, const float* lo, const float* st,
                        const float* top, const float* hs, int64_t n_rows, int64_t k, int64_t b0, float* dwb,
                        float* dw_lo, int64_t lddw, int32_t* moved, cudaStream_t stream) {
  if (two_rows_per_lane(n_rows))
    return launch_refine_as<2>(gb, ldg, len, c, lo, st, top, hs, n_rows, k, b0, dwb, dw_lo, lddw, moved, stream);
  return launch_refine_as<1>(gb, ldg, len, c, lo, st, top, hs, n_rows, k, b0, dwb, dw_lo, lddw, moved, stream);
}

}  // namespace
}  // namespace hi2

extern "C" int hi2_refine_block(const float* gb, int len, float* c, const float* lo,
                                const float* st, const float* top, const float* hs, int64_t n_rows,
                                int64_t k, int64_t b0, float* dwb, void* stream) {
  using namespace hi2;
  HI2_REQUIRE(k > 0 && k % 16 == 0, "refine_block: k must be a positive multiple of 16");
  HI2_REQUIRE(len > 0 && len <= LMAX && len % 16 == 0, "refine_block: block length must be 16..128");
  HI2_REQUIRE(b0 >= 0 && b0 % 16 == 0 && b0 + len <= k, "refine_block: block outside the row");
  if (n_rows == 0) return HI2_OK;
  HI2_REQUIRE(gb && c && lo && st && top && hs && dwb, "refine_block: null pointer");
  HI2_REQUIRE(aligned16(gb) && aligned16(c) && aligned16(lo) && aligned16(st) && aligned16(hs) &&
                  aligned16(dwb),
              "refine_block: buffers must be 16-byte aligned");
  return launch_refine_block(gb, len, len, c, lo, st, top, hs, n_rows, k, b0, dwb, nullptr, len, nullptr,
                             static_cast<cudaStream_t>(stream));
}

extern "C" int hi2_refine_block_in_place(const float* g, int len, float* c, const float* lo, const float* st,
                                         const float* top, const float* hs, int64_t n_rows, int64_t k,
                                         int64_t b0, float* dw_hi, float* dw_lo, int64_t lddw, void* stream) {
  return hi2_refine_sweep_block(g, len, c, lo, st, top, hs, n_rows, k, b0, dw_hi, dw_lo, lddw, nullptr, stream);
}

extern "C" int hi2_refine_sweep_block(const float* g, int len, float* c, const float* lo, const float* st,
                                      const float* top, const float* hs, int64_t n_rows, int64_t k, int64_t b0,
                                      float* dw_hi, float* dw_lo, int64_t lddw, int32_t* moved, void* stream) {
  using namespace hi2;
  HI2_REQUIRE(k > 0 && k % 16 == 0, "refine_block_in_place: k must be a positive multiple of 16");
  HI2_REQUIRE(len > 0 && len <= LMAX && len % 16 == 0, "refine_block_in_place: block length must be 16..128");
  HI2_REQUIRE(b0 >= 0 && b0 % 16 == 0 && b0 + len <= k, "refine_block_in_place: block outside the row");
  HI2_REQUIRE(lddw >= len && lddw % 4 == 0, "refine_block_in_place: lddw must cover the block and be a multiple of 4");
  if (n_rows == 0) return HI2_OK;
  HI2_REQUIRE(g && c && lo && st && top && hs && dw_hi && dw_lo, "refine_block_in_place: null pointer");
  HI2_REQUIRE(aligned16(g) && aligned16(c) && aligned16(lo) && aligned16(st) && aligned16(hs) &&
                  aligned16(dw_hi) && aligned16(dw_lo),
              "refine_block_in_place: buffers must be 16-byte aligned");
  return launch_refine_block(g + b0, k, len, c, lo, st, top, hs, n_rows, k, b0, dw_hi, dw_lo, lddw, moved,
                             static_cast<cudaStream_t>(stream));
}

extern "C" int hi2_refine_prepare(const float* w, int64_t ldw, const uint8_t* codes, const uint8_t* params,
                                  const uint16_t* consts, int block, int64_t n_rows, int64_t k, float* c, float* lo_x,
                                  float* st_x, float* e, float* e_lo, void* stream) {
  using namespace hi2;
  HI2_REQUIRE(block == 16 || block == 32 || block == 64, "refine_prepare: block must be 16, 32 or 64");
  HI2_REQUIRE(k > 0 && k % block == 0, "refine_prepare: k must be a multiple of the block");
  if (n_rows == 0) return HI2_OK;
  HI2_REQUIRE(w && codes && params && consts && c && lo_x && st_x && e, "refine_prepare: null pointer");
  HI2_REQUIRE(aligned16(w) && ldw % 4 == 0 && ldw >= k && (reinterpret_cast<uintptr_t>(codes) & 3u) == 0 &&
                  (reinterpret_cast<uintptr_t>(params) & 1u) == 0 && aligned16(c) && aligned16(lo_x) && aligned16(st_x) &&
                  aligned16(e) && (e_lo == nullptr || aligned16(e_lo)),
              "refine_prepare: alignment or ldw");
  const dim3 grid((unsigned)(n_rows < 65536 ? n_rows : 65536), (unsigned)ceil_div(k, (int64_t)1024));
  refine_prepare_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      w, ldw, codes, params, consts, block == 16 ? 4 : block == 32 ? 5 : 6, n_rows, k, c, lo_x, st_x, e, e_lo);
  return check_launch("refine_prepare");
}

extern "C" int hi2_refine_sweep(float* g, float* c, const float* lo, const float* st, const float* top, const float* hs,
                                const float* hs_split, float* moves, int64_t n_rows, int64_t k, int64_t width, int last,
                                int32_t* moved, int32_t* status, void* stream) {
  using namespace hi2;
  HI2_REQUIRE(k > 0 && k % 16 == 0, "refine_sweep: k must be a positive multiple of 16");
  HI2_REQUIRE(width >= LMAX && width % LMAX == 0, "refine_sweep: width must be a multiple of 128");
  if (n_rows == 0) return HI2_OK;
  HI2_REQUIRE(g && c && lo && st && top && hs && moves && (hs_split == nullptr || status), "refine_sweep: null pointer");
  HI2_REQUIRE(aligned16(g) && aligned16(c) && aligned16(lo) && aligned16(st) && aligned16(hs) && aligned16(moves) &&
                  (hs_split == nullptr || aligned16(hs_split)),
              "refine_sweep: buffers must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  ChainGraph chain(s, 2 * ceil_div(k, (int64_t)LMAX));
  auto enqueue = [&]() -> int {
    int rc;
    if (hs_split == nullptr) {  // fp32 FMA products, block by block
      for (int64_t b0 = 0; b0 < k; b0 += LMAX) {
        const int64_t b1 = b0 + LMAX < k ? b0 + LMAX : k, first = last ? b1 : 0;
        const int len = (int)(b1 - b0);
        rc = launch_refine_block(g + b0, k, len, c, lo, st, top, hs, n_rows, k, b0, moves, nullptr, len, moved, s);
        if (rc != HI2_OK) return rc;
        if (first >= k) continue;
        GemmArgs<float, float, float> p;
        p.m = n_rows, p.n = k - first, p.kk = len, p.alpha = 1.0f, p.beta = 1.0f;
        p.a = moves, p.lda = len, p.b = hs + b0 * k + first, p.ldb = k, p.c = g + first, p.ldc = k, p.flags = 0;
        rc = launch_gemm_async<float, 8, 8, 16>(false, false, p, s, "refine_sweep");
        if (rc != HI2_OK) return rc;
      }
      return HI2_OK;
    }
    // Tensor-core products.  After a block the rest of its group needs its moves now; the columns outside
    // the group take the whole group's in one product; the group's own columns at or before each block
    // are needed by the next sweep only.  hs is symmetric: its rows are the K-major right operand.
    const int64_t ldm = width < k ? width : k;
    float *hi = moves, *lo_part = moves + n_rows * ldm;
    int* word = reinterpret_cast<int*>(status);
    auto product = [&](int64_t b0, int64_t b1, int64_t g0, int64_t c0, int64_t c1) -> int {  // g[:, c0:c1] += moves of [b0, b1)
      if (c0 >= c1) return HI2_OK;
      return launch_gemm_tc2(n_rows, c1 - c0, b1 - b0, hi + (b0 - g0), lo_part + (b0 - g0), ldm, hs_split + c0 * k + b0,
                             hs_split + k * k + c0 * k + b0, k, g + c0, k, GT_ADD, word, s);
    };
    for (int64_t g0 = 0; g0 < k; g0 += width) {
      const int64_t g1 = g0 + width < k ? g0 + width : k;
      for (int64_t b0 = g0; b0 < g1; b0 += LMAX) {
        const int64_t b1 = b0 + LMAX < g1 ? b0 + LMAX : g1;
        rc = launch_refine_block(g + b0, k, (int)(b1 - b0), c, lo, st, top, hs, n_rows, k, b0, hi + (b0 - g0),
                                 lo_part + (b0 - g0), ldm, moved, s);
        if (rc != HI2_OK) return rc;
        if ((rc = product(b0, b1, g0, b1, g1)) != HI2_OK) return rc;
      }
      if (width == LMAX) {  // groups of one block: the whole update in one product
        if ((rc = product(g0, g1, g0, last ? g1 : 0, k)) != HI2_OK) return rc;
        continue;
      }
      if (!last && (rc = product(g0, g1, g0, 0, g0)) != HI2_OK) return rc;
      if ((rc = product(g0, g1, g0, g1, k)) != HI2_OK) return rc;
      for (int64_t b0 = g0; b0 < g1 && !last; b0 += LMAX)
        if ((rc = product(b0, g1, g0, b0, b0 + LMAX < g1 ? b0 + LMAX : g1)) != HI2_OK) return rc;
    }
    return HI2_OK;
  };
  return chain.finish(enqueue(), "refine_sweep");
}
