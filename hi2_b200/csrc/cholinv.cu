// Damped inverse factor (hi2/hessian.py:71-86): the upper-triangular U with
// U^T U = (hs + lam I)^-1.
//
// The reference factorises, inverts and factorises again.  The same U has a closed form: with J
// the index reversal, J (hs + lam I) J = L L^T (L lower) gives U = J L^-1 J.  So one Cholesky
// factorisation and one triangular inverse suffice, and both come out of one recursion on the
// reversed matrix A (fp32, lower part):
//
//   F(A):  split A = [A11 . ; A21 A22]
//          (X11) = F(A11)                      X11 = L11^-1
//          W     = A21 X11^T                   (= L21)
//          A22  -= W W^T
//          T     = W X11
//          (X22) = F(A22)
//          X21   = -X22 T
//
// The bottom of the recursion is a block of 128 (base_kernel: two 64-wide leaves in fp64 and the four
// products between them, one launch); above it every step is a matrix product, product_kernel (fp32
// FMA) up to sides of 1024 and three TF32 tensor-core products (lazy_tc.cu) from there on, with
// triangular operands expressed as k-ranges.  W is kept in the X21 slot and T in the A21 slot, so the
// scratch is 2 K^2 floats.  Measured before (a launch per leaf and per 64-wide product) and after, the
// whole factor: K = 1024 2.4 -> 0.53 ms, 4096 9.9 -> 2.5 ms, 11008 33.8 -> 11.5 ms; what is left is the
// chain of K / 128 base blocks (32 us each) and, at 11008, 5.4 ms of tensor-core products.
// Precision: the reference's own path is fp32 LAPACK; measured against an fp64 solution on
// calibration-like Hessians (K = 1024..2048, condition 3e3..8e4) this recursion with fp32
// products is as close to the truth as the reference is (1.0e-5 vs 1.5e-5 of max|U| at condition
// 5e3, 3e-4 vs 1.4e-3 at 8e4), and fp64 products would not bring it closer to the REFERENCE,
// whose own rounding dominates the difference either way.  A non-positive pivot does not trap:
// the leaf records its index in *info, carries on with a unit pivot, and the host retries with
// more damping.
#include "gemm.cuh"

namespace hi2 {
// lazy_tc.cu
int launch_gemm_tc(int64_t m, int64_t n, int64_t kk, const float* a_hi, const float* a_lo, const float* b_hi,
                   const float* b_lo, int64_t ldk, float* c, int64_t ldc, int flags, int* status,
                   cudaStream_t stream);
int launch_split_block(const float* x, int64_t ldx, int64_t rows, int64_t cols, float* hi, float* lo,
                       int64_t ldo, bool transposed, bool lower, cudaStream_t stream);
namespace {

constexpr int NB = 64;     // a leaf: factorised and inverted in fp64 registers
constexpr int BASE = 128;  // the bottom of the recursion: two leaves and the four products between them
constexpr int LDF = BASE + 4;  // rows 4 banks apart: 128-bit reads of eight neighbouring rows hit every bank once
// doubles of a leaf's exchange buffers: panel columns [64][9], panel rows [8][66], update vectors [64][12],
// and one 8 x 8 block for each of two warps
constexpr int LEAF_PCOL = 0, LEAF_PROW = LEAF_PCOL + NB * 9, LEAF_G = LEAF_PROW + 8 * 66,
              LEAF_M = LEAF_G + NB * 12, LEAF_DOUBLES = LEAF_M + 2 * 64;
constexpr size_t BASE_SMEM = (size_t)LEAF_DOUBLES * sizeof(double) + (size_t)2 * BASE * LDF * sizeof(float);

// A[i][j] = hs[k-1-i][k-1-j] for j <= i (+ lam on the diagonal, added in fp32 as the reference does).
// Nothing reads above the diagonal of A, so only the lower half is moved; four columns per thread
// (VEC: k is a multiple of 4, so the reversed quads are aligned too).
template <bool VEC>
__global__ void __launch_bounds__(256)
reverse_damp_kernel(const float* __restrict__ hs, const float* __restrict__ lam, int64_t k, int64_t ld,
                    float* __restrict__ a) {
  const int64_t i = blockIdx.x, j = ((int64_t)blockIdx.y * 256 + threadIdx.x) * 4;
  if (j > i) return;
  const float* src = hs + (k - 1 - i) * k;
  float v[4];
  if (VEC) {
    const float4 q = *reinterpret_cast<const float4*>(src + (k - 4 - j));
    v[0] = q.w, v[1] = q.z, v[2] = q.y, v[3] = q.x;
  } else {
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = j + t < k ? src[k - 1 - j - t] : 0.0f;
  }
  if (i - j < 4) {
    const float damp = *lam;
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (j + t == i) v[t] = v[t] + damp;
  }
  *reinterpret_cast<float4*>(a + i * ld + j) = make_float4(v[0], v[1], v[2], v[3]);
}

// u[i][j] = x[k-1-i][k-1-j] for j >= i, zero below the diagonal (the upper half of x is not read).
template <bool VEC>
__global__ void __launch_bounds__(256)
reverse_store_kernel(const float* __restrict__ x, int64_t k, int64_t ld, float* __restrict__ u) {
  const int64_t i = blockIdx.x, j = ((int64_t)blockIdx.y * 256 + threadIdx.x) * 4;
  if (j >= k) return;
  const float* src = x + (k - 1 - i) * ld;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (j + 3 >= i) {
    if (VEC) {
      const float4 q = *reinterpret_cast<const float4*>(src + (k - 4 - j));
      v[0] = q.w, v[1] = q.z, v[2] = q.y, v[3] = q.x;
    } else {
#pragma unroll
      for (int t = 0; t < 4; ++t) v[t] = j + t < k ? src[k - 1 - j - t] : 0.0f;
    }
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (j + t < i) v[t] = 0.0f;
  }
  if (VEC) {
    *reinterpret_cast<float4*>(u + i * k + j) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (j + t < k) u[i * k + j + t] = v[t];
  }
}

// 1 / sqrt(v) in fp64 for v in [1e-300, 1e300]: the hardware's estimate y (20 bits), then
// y (1 - r)^(-1/2) with r = 1 - v y^2 as y (1 + r / 2 + 3 r^2 / 8); the next term is below 2^-57.
__device__ __forceinline__ double inv_sqrt(double v) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
  const double r = fma(-(v * y), y, 1.0);
  return fma(y * r, fma(r, 0.375, 0.5), y);
}

// L of an 8 x 8 diagonal block (lower part at d, rows 9 apart) one pivot at a time with the plain root
// and quotient, for blocks with a pivot that is not positive (recorded in *info, taken as one) or
// outside the range of inv_sqrt.  One lane; out: L below the diagonal, 1 / L_jj on it, rows 8 apart.
__device__ __noinline__ void factor8_careful(const double* d, double* out, int32_t* info, int32_t pivot0, bool report) {
  for (int i = 0; i < 8; ++i)
    for (int j = 0; j <= i; ++j) out[i * 8 + j] = d[i * 9 + j];
  for (int j = 0; j < 8; ++j) {
    double piv = out[j * 8 + j];
    if (!(piv > 0.0)) {  // also catches NaN
      if (report) atomicCAS(info, 0, pivot0 + j + 1);
      piv = 1.0;
    }
    const double r = 1.0 / sqrt(piv);
    for (int i = j + 1; i < 8; ++i) out[i * 8 + j] *= r;
    for (int i = j + 1; i < 8; ++i)
      for (int q = j + 1; q <= i; ++q) out[i * 8 + q] = fma(-out[i * 8 + j], out[q * 8 + j], out[i * 8 + q]);
    out[j * 8 + j] = r;
  }
}

// c[8, 8] += a[8, 4] b[4, 8] in fp64 on the tensor cores, skipped where `on` is zero (lane l holds a[l / 4][l % 4],
// b[l % 4][l / 4], c[l / 4][2 (l % 4)] and its right neighbour)
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b, int on) {
  asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %4, 0;\n\t"
      "@p mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n\t}"
      : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b), "r"(on));
}

// X = L^-1 of the 64 x 64 block at (o, o) of `sa` (lower part, L L^T = A), written to the same place
// of `sx` with zeros above the diagonal.  Rows at or past n_loc are taken from the identity.  256
// threads; fp64 throughout, rounded to fp32 once at the end.
//
// Elimination on [A | I] in place, eight columns a panel: after a panel the eliminated columns hold
// rows of X (the identity's part), the others the Schur complement, so one 64 x 64 array serves
// factorisation and inversion and L itself is never kept.  The array lives in registers: warp w
// holds rows 8 w .. 8 w + 7 as eight 8 x 8 tiles in the layout of the fp64 tensor-core product.  Per
// panel: its columns and rows are published in shared memory; two warps factorise the 8 x 8 diagonal
// block (all lanes alike, no exchange) and lane i solves for row i of L's panel, or for column i of
// X's panel where column i is already eliminated; then the warps below the panel apply the rank-8
// update, two tensor-core products per tile.  Two barriers per panel, sixteen per leaf; the panel loop
// is kept rolled because unrolled code runs once and waits for instruction fetch.
// The time is the chain of 32 pairs of pivots.  Base block of 128, us: one column per barrier and the
// inversion as a second chain, one launch per product 182; this with branches in the pivot chain 43;
// without 34; with the update on the fp64 tensor cores (its operands from shared memory bound it: a
// thread's 4 x 4 tile reads 64 doubles for 80 products) and without an explicit inverse of the diagonal
// block 32.
__device__ __forceinline__ void leaf_inverse(const float* sa, float* sx, int o, int n_loc, double* ex, int32_t* info,
                                             int32_t pivot0) {
  double* pcol = ex + LEAF_PCOL;
  double* prow = ex + LEAF_PROW;
  double* gv = ex + LEAF_G;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, q = lane & 3;
  const int i = 8 * warp + r;  // this lane's row
  double c[8][2];
#pragma unroll
  for (int t = 0; t < 8; ++t)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int j = 8 * t + 2 * q + e;
      c[t][e] = i >= n_loc ? (i == j ? 1.0 : 0.0) : (j <= i ? (double)sa[(o + i) * LDF + o + j] : 0.0);
    }
#pragma unroll 1
  for (int p = 0; p < NB / 8; ++p) {
    const int j0 = 8 * p;
    if (warp >= p) {
#pragma unroll
      for (int t = 0; t < 8; ++t)
        if (t == p) {
          pcol[i * 9 + 2 * q] = c[t][0], pcol[i * 9 + 2 * q + 1] = c[t][1];
          c[t][0] = c[t][1] = 0.0;  // from here on the column holds X
        }
    }
    if (warp == p) {
#pragma unroll
      for (int t = 0; t < 8; ++t)
        if (t < p) prow[r * 66 + 8 * t + 2 * q] = c[t][0], prow[r * 66 + 8 * t + 2 * q + 1] = c[t][1];
    }
    __syncthreads();
    if (tid < NB) {
      double d[8][8], ri[8], w[8];
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = 0; b <= a; ++b) d[a][b] = pcol[(j0 + a) * 9 + b];
      // lane tid: row tid of the panel below the diagonal block, else column tid of the panel's rows
      const bool row = tid >= j0 + 8;
#pragma unroll
      for (int s = 0; s < 8; ++s)
        w[s] = row ? pcol[tid * 9 + s] : (tid < j0 ? prow[s * 66 + tid] : (s == tid - j0 ? 1.0 : 0.0));
      // Pivots in pairs: the second pivot of a pair is det / p0, so both reciprocal roots are taken side
      // by side and the chain of 64 becomes one of 32.  Whether every pivot was positive is asked once
      // at the end: a branch per pivot would stand in the chain.
      bool fine = true;
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        const double p0 = d[j][j], e = d[j + 1][j], det = fma(-e, e, p0 * d[j + 1][j + 1]);
        fine = fine && p0 > 1e-150 && p0 < 1e150 && det > 1e-300 && det < 1e300;  // false for NaN
        const double r0 = inv_sqrt(p0), r1 = inv_sqrt(det) * (p0 * r0), l10 = e * r0;
        ri[j] = r0, ri[j + 1] = r1;
        d[j + 1][j] = l10;
#pragma unroll
        for (int a = j + 2; a < 8; ++a) {
          d[a][j] *= r0;
          d[a][j + 1] = fma(-d[a][j], l10, d[a][j + 1]) * r1;
        }
#pragma unroll
        for (int a = j + 2; a < 8; ++a)
#pragma unroll
          for (int b = j + 2; b <= a; ++b) d[a][b] = fma(-d[a][j + 1], d[b][j + 1], fma(-d[a][j], d[b][j], d[a][b]));
      }
      if (!fine) {  // the same for all 64 lanes
        double* own = ex + LEAF_M + warp * 64;
        if (lane == 0) factor8_careful(pcol + j0 * 9, own, info, pivot0 + j0, tid == 0);
        __syncwarp();
#pragma unroll
        for (int a = 0; a < 8; ++a) {
#pragma unroll
          for (int b = 0; b < a; ++b) d[a][b] = own[a * 8 + b];
          ri[a] = own[a * 8 + a];
        }
        __syncwarp();
      }
#pragma unroll
      for (int s = 0; s < 8; ++s) {  // y = L^-1 w
        w[s] *= ri[s];
#pragma unroll
        for (int a = s + 1; a < 8; ++a) w[a] = fma(-d[a][s], w[s], w[a]);
        gv[tid * 12 + s] = w[s];
      }
    }
    __syncthreads();
    // Element (i, j) loses the product of vector i (a row of L) and vector j (a row of L, or a column of
    // X for the columns eliminated so far).
    if (warp > p) {
      const double a0 = -gv[i * 12 + q], a1 = -gv[i * 12 + 4 + q];
      double b0[8], b1[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) b0[t] = gv[(8 * t + r) * 12 + q], b1[t] = gv[(8 * t + r) * 12 + 4 + q];
#pragma unroll
      for (int t = 0; t < 8; ++t) dmma(c[t], a0, b0[t], t <= warp);
#pragma unroll
      for (int t = 0; t < 8; ++t) dmma(c[t], a1, b1[t], t <= warp);
    } else if (warp == p) {  // the panel's rows of X are final
#pragma unroll
      for (int t = 0; t < 8; ++t)
        if (t <= p) c[t][0] = gv[(8 * t + 2 * q) * 12 + r], c[t][1] = gv[(8 * t + 2 * q + 1) * 12 + r];
    }
  }
#pragma unroll
  for (int t = 0; t < 8; ++t)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int j = 8 * t + 2 * q + e;
      sx[(o + i) * LDF + o + j] = j <= i ? (float)c[t][e] : 0.0f;
    }
}

__device__ __forceinline__ float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float dot4(float4 a, float4 b, float acc) {
  acc = fmaf(a.x, b.x, acc);
  acc = fmaf(a.y, b.y, acc);
  acc = fmaf(a.z, b.z, acc);
  return fmaf(a.w, b.w, acc);
}

// F of one diagonal block of n <= 128 rows: two leaves and the four 64 x 64 x 64 products between
// them (fp32 FMA), everything in shared memory, one thread block of 256 threads.  In global memory
// only x changes (zeros above the diagonal of the block included).  As two leaf launches and four
// product launches of one thread block each this cost 182 us.
__global__ void __launch_bounds__(256, 1)
base_kernel(const float* __restrict__ a, float* __restrict__ x, int64_t ld, int64_t off, int n, int32_t* info) {
  extern __shared__ double base_smem[];
  chain_wait();
  float* sa = reinterpret_cast<float*>(base_smem + LEAF_DOUBLES);
  float* sx = sa + BASE * LDF;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const float* src = a + off * ld + off;
  for (int idx = tid; idx < BASE * BASE / 4; idx += 256) {
    const int i = idx >> 5, j = (idx & 31) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n && j <= i) v = *reinterpret_cast<const float4*>(src + (int64_t)i * ld + j);
    *reinterpret_cast<float4*>(sa + i * LDF + j) = v;  // past the diagonal: not read
    *reinterpret_cast<float4*>(sx + i * LDF + j) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  float* w = sx + NB * LDF;  // W = A21 X11^T, in the place of X21
  float* a21 = sa + NB * LDF;
  float* a22 = a21 + NB;
  float acc[4][4];
#pragma unroll 1
  for (int o = 0; o < n; o += NB) {  // one copy of the leaf's code serves both
    leaf_inverse(sa, sx, o, min(n - o, NB), base_smem, info, (int32_t)off + o);
    __syncthreads();
    if (o > 0 || n <= NB) break;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[r][b] = 0.0f;
#pragma unroll
    for (int kb = 0; kb < 4; ++kb)  // X11[j][k] is zero for k > j
      for (int k = 16 * kb; k < 16 * kb + 16; k += 4) {
        float4 av[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) av[r] = lds4(a21 + (ty + 16 * r) * LDF + k);
#pragma unroll
        for (int b = kb; b < 4; ++b) {
          const float4 bv = lds4(sx + (tx + 16 * b) * LDF + k);
#pragma unroll
          for (int r = 0; r < 4; ++r) acc[r][b] = dot4(av[r], bv, acc[r][b]);
        }
      }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int b = 0; b < 4; ++b) w[(ty + 16 * r) * LDF + tx + 16 * b] = acc[r][b];
    __syncthreads();
    // A22 -= W W^T (lower part)
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[r][b] = 0.0f;
    for (int k = 0; k < NB; k += 4) {
      float4 av[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) av[r] = lds4(w + (ty + 16 * r) * LDF + k);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const float4 bv = lds4(w + (tx + 16 * b) * LDF + k);
#pragma unroll
        for (int r = b; r < 4; ++r) acc[r][b] = dot4(av[r], bv, acc[r][b]);
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int b = 0; b <= r; ++b) a22[(ty + 16 * r) * LDF + tx + 16 * b] -= acc[r][b];
    // T = W X11, in the place of A21; columns 4 tx + b here
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[r][b] = 0.0f;
    for (int k = 0; k < NB; k += 4) {
      float4 av[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) av[r] = lds4(w + (ty + 16 * r) * LDF + k);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float4 bv = lds4(sx + (k + t) * LDF + 4 * tx);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float e = t == 0 ? av[r].x : t == 1 ? av[r].y : t == 2 ? av[r].z : av[r].w;
          acc[r][0] = fmaf(e, bv.x, acc[r][0]);
          acc[r][1] = fmaf(e, bv.y, acc[r][1]);
          acc[r][2] = fmaf(e, bv.z, acc[r][2]);
          acc[r][3] = fmaf(e, bv.w, acc[r][3]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
      *reinterpret_cast<float4*>(a21 + (ty + 16 * r) * LDF + 4 * tx) =
          make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    __syncthreads();
  }
  if (n > NB) {
    // X21 = -X22 T; X22[i][k] is zero for k > i
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[r][b] = 0.0f;
#pragma unroll
    for (int kb = 0; kb < 4; ++kb)
      for (int k = 16 * kb; k < 16 * kb + 16; k += 4) {
        float4 av[4];
#pragma unroll
        for (int r = kb; r < 4; ++r) av[r] = lds4(w + NB + (ty + 16 * r) * LDF + k);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float4 bv = lds4(a21 + (k + t) * LDF + 4 * tx);
#pragma unroll
          for (int r = kb; r < 4; ++r) {
            const float e = t == 0 ? av[r].x : t == 1 ? av[r].y : t == 2 ? av[r].z : av[r].w;
            acc[r][0] = fmaf(e, bv.x, acc[r][0]);
            acc[r][1] = fmaf(e, bv.y, acc[r][1]);
            acc[r][2] = fmaf(e, bv.z, acc[r][2]);
            acc[r][3] = fmaf(e, bv.w, acc[r][3]);
          }
        }
      }
#pragma unroll
    for (int r = 0; r < 4; ++r)
      *reinterpret_cast<float4*>(w + (ty + 16 * r) * LDF + 4 * tx) =
          make_float4(-acc[r][0], -acc[r][1], -acc[r][2], -acc[r][3]);
    __syncthreads();
  }
  chain_next();
  float* dst = x + off * ld + off;
  for (int idx = tid; idx < n * (BASE / 4); idx += 256) {
    const int i = idx >> 5, j = (idx & 31) * 4;
    if (j < n) *reinterpret_cast<float4*>(dst + (int64_t)i * ld + j) = lds4(sx + i * LDF + j);
  }
}

// ---------------------------------------------------------------------------------------------
// Products of the levels between a base block and the tensor cores (n2 below 1024, n1 up to 1152):
//
//   C[m, n] = or -= A[m, kk] . B,   B given as Bt[n, kk] (TRANS) or as B[kk, n]
//
// These are a few small tiles on a dependency chain, so the time is launch, memory latency and the
// length of a tile's own reduction, not throughput: a thread block takes a 32 x 32 tile and its four
// groups of two warps each sum a quarter of the reduction (32 of every 128 values of k), added in
// a fixed order at the end.  At 128 x 128 x 128 that is 16 thread blocks of 32 steps where 128 x 128
// tiles were one block of 128 steps: 4 us against 19 us.  The four sums also keep every fp32 chain at
// a quarter of the reduction (at most 288 values; one chain per dot product costs a decimal digit on
// rank-deficient, damped Hessians).  Two independent products can share a launch (blockIdx.z).
constexpr int PT = 32, P_GROUPS = 4, P_STEP = 32, P_STAGES = 3, P_LD = P_STEP + 4;
constexpr int P_TILE = PT * P_LD;                               // floats of one operand tile
constexpr int P_STAGE = P_GROUPS * 2 * P_TILE;                  // floats of one stage
constexpr size_t P_SMEM = (size_t)P_STAGES * P_STAGE * sizeof(float);

struct ProductJob {
  const float* a;
  const float* b;
  float* c;
  int m, n, kk;
  int flags;       // GEMM_* of gemm.cuh
  int trans;       // B is Bt [n, kk]
  int subtract;    // C -= instead of C =
  int negate;      // C = -(A B)
};

__device__ __forceinline__ void copy16(float* dst, const float* src, int floats) {
  const int bytes = floats >= 4 ? 16 : (floats > 0 ? floats * 4 : 0);  // the rest is zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes) : "memory");
}

__global__ void __launch_bounds__(256, 2)
product_kernel(const ProductJob job0, const ProductJob job1, int64_t ld) {
  extern __shared__ __align__(16) float product_smem[];
  chain_wait();
  const ProductJob& p = blockIdx.z ? job1 : job0;
  const int m0 = blockIdx.y * PT, n0 = blockIdx.x * PT;
  if (m0 >= p.m || n0 >= p.n) return;
  if ((p.flags & GEMM_LOWER_OUT) && n0 > m0) return;
  const int tid = threadIdx.x, g = tid >> 6, lt = tid & 63, tx = lt & 7, ty = lt >> 3;
  int k_lo = 0, k_hi = p.kk;
  if (p.flags & GEMM_KA_LE_I) k_hi = min(k_hi, m0 + PT);
  if (p.flags & GEMM_KB_LE_J) k_hi = min(k_hi, n0 + PT);
  if (p.flags & GEMM_KB_GE_J) k_lo = n0;  // a multiple of 32
  const int rounds = (k_hi - k_lo + P_GROUPS * P_STEP - 1) / (P_GROUPS * P_STEP);

  auto issue = [&](int r) {
    float* as = product_smem + (r % P_STAGES) * P_STAGE + g * 2 * P_TILE;
    float* bs = as + P_TILE;
    const int k0 = k_lo + (r * P_GROUPS + g) * P_STEP;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int idx = lt + s * 64, row = idx >> 3, q = (idx & 7) * 4;
      const int left = m0 + row < p.m ? k_hi - (k0 + q) : 0;
      copy16(as + row * P_LD + q, left > 0 ? p.a + (int64_t)(m0 + row) * ld + k0 + q : p.a, left);
      if (p.trans) {
        const int leftb = n0 + row < p.n ? k_hi - (k0 + q) : 0;
        copy16(bs + row * P_LD + q, leftb > 0 ? p.b + (int64_t)(n0 + row) * ld + k0 + q : p.b, leftb);
      } else {
        const int leftb = k0 + row < k_hi ? p.n - (n0 + q) : 0;
        copy16(bs + row * P_LD + q, leftb > 0 ? p.b + (int64_t)(k0 + row) * ld + n0 + q : p.b, leftb);
      }
    }
  };
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
#pragma unroll
  for (int s = 0; s < P_STAGES - 1; ++s) {
    if (s < rounds) issue(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int r = 0; r < rounds; ++r) {
    asm volatile("cp.async.wait_group %0;" ::"n"(P_STAGES - 2) : "memory");
    __syncthreads();  // round r has landed for everyone; the stage of round r - 1 is free
    if (r + P_STAGES - 1 < rounds) issue(r + P_STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* as = product_smem + (r % P_STAGES) * P_STAGE + g * 2 * P_TILE;
    const float* bs = as + P_TILE;
    if (p.trans) {  // rows ty + 8 i, columns tx + 8 j
#pragma unroll
      for (int k = 0; k < P_STEP; k += 4) {
        float4 av[4], bv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) av[i] = lds4(as + (ty + 8 * i) * P_LD + k), bv[i] = lds4(bs + (tx + 8 * i) * P_LD + k);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = dot4(av[i], bv[j], acc[i][j]);
      }
    } else {  // rows ty + 8 i, columns 4 tx + j
#pragma unroll
      for (int k = 0; k < P_STEP; k += 4) {
        float4 av[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) av[i] = lds4(as + (ty + 8 * i) * P_LD + k);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float4 bv = lds4(bs + (k + t) * P_LD + 4 * tx);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float e = t == 0 ? av[i].x : t == 1 ? av[i].y : t == 2 ? av[i].z : av[i].w;
            acc[i][0] = fmaf(e, bv.x, acc[i][0]);
            acc[i][1] = fmaf(e, bv.y, acc[i][1]);
            acc[i][2] = fmaf(e, bv.z, acc[i][2]);
            acc[i][3] = fmaf(e, bv.w, acc[i][3]);
          }
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  chain_next();
  float* part = product_smem + g * P_TILE;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) part[(ty + 8 * i) * P_LD + (p.trans ? tx + 8 * j : 4 * tx + j)] = acc[i][j];
  __syncthreads();
  const int row = tid >> 3, col = (tid & 7) * 4;
  if (m0 + row >= p.m || n0 + col >= p.n) return;
  const float* src = product_smem + row * P_LD + col;
  float v[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    v[t] = (src[t] + src[P_TILE + t]) + (src[2 * P_TILE + t] + src[3 * P_TILE + t]);
    if (p.negate) v[t] = -v[t];
  }
  // rows are padded to whole quads, so the last quad of a row may run into the padding
  float4* dst = reinterpret_cast<float4*>(p.c + (int64_t)(m0 + row) * ld + n0 + col);
  if (p.subtract) {
    const float4 old = *dst;
    v[0] = old.x - v[0], v[1] = old.y - v[1], v[2] = old.z - v[2], v[3] = old.w - v[3];
  }
  *dst = make_float4(v[0], v[1], v[2], v[3]);
}

int launch_products(const ProductJob& j0, const ProductJob* j1, int64_t ld, cudaStream_t stream) {
  const ProductJob& other = j1 ? *j1 : j0;
  dim3 grid((unsigned)ceil_div(j0.n > other.n ? j0.n : other.n, PT), (unsigned)ceil_div(j0.m > other.m ? j0.m : other.m, PT),
            j1 ? 2 : 1);
  launch_link(product_kernel, grid, 256, P_SMEM, stream, j0, other, ld);
  return check_launch("inverse_factor product");
}

struct Plan {
  float* a;
  float* x;
  int64_t ld;    // leading dimension of a and x: k rounded up to whole 16-byte pieces
  float* split;  // TF32 parts of the operands of one tensor-core product (4 n1^2 floats)
  int* status;   // raised by a tensor-core product whose bounded wait ran out
  int64_t k;
  int32_t* info;
  cudaStream_t stream;
};

constexpr int GT_KB_LE_J = 1, GT_KB_GE_J = 2, GT_KA_LE_I = 4, GT_LOWER_OUT = 8, GT_NEGATE = 16, GT_ADD = 32;

// Products at least this large on both output sides go to the tensor cores (3xTF32, fp32-grade);
// below it a 128 x 256 tile grid no longer fills the SMs and the FMA kernel is as fast.
#ifndef HI2_FACTOR_TC_MIN
#define HI2_FACTOR_TC_MIN 1024
#endif

// The upper part of a split: whole base blocks, so that every base block but the last one is full.
int64_t top_half(int64_t n) { return ((ceil_div(n, (int64_t)BASE) + 1) / 2) * BASE; }
int64_t padded(int64_t k) { return (k + 3) / 4 * 4; }
size_t split_floats(int64_t k) {
  const int64_t n1 = top_half(k);
  return k >= 2 * HI2_FACTOR_TC_MIN ? (size_t)(4 * n1 * n1) : 0;
}
__global__ void merge_status_kernel(const int* status, int32_t* info) {
  if (*status != 0) *info = -1;
}

// Launches of F on n rows, for the chain's choice between a graph and plain launches.
int64_t chain_length(int64_t n) {
  if (n <= BASE) return 1;
  const int64_t n1 = top_half(n), n2 = n - n1;
  return chain_length(n1) + chain_length(n2) + (n2 >= HI2_FACTOR_TC_MIN ? 13 : 3);
}

int factor(const Plan& pl, int64_t off, int64_t n) {
  const int64_t ld = pl.ld;
  if (n <= BASE) {
    launch_link(base_kernel, 1, 256, BASE_SMEM, pl.stream, pl.a, pl.x, ld, off, (int)n, pl.info);
    return check_launch("inverse_factor base");
  }
  const int64_t n1 = top_half(n), n2 = n - n1;
  int rc = factor(pl, off, n1);
  if (rc != HI2_OK) return rc;
  float* a21 = pl.a + (off + n1) * ld + off;
  float* a22 = pl.a + (off + n1) * ld + off + n1;
  float* x11 = pl.x + off * ld + off;
  float* x21 = pl.x + (off + n1) * ld + off;
  float* x22 = pl.x + (off + n1) * ld + off + n1;
  if (n2 >= HI2_FACTOR_TC_MIN && pl.split != nullptr) {
    // Tensor-core path.  Operands are split into TF32 parts first (K-major; the right-hand
    // operands of T = W X11 and X21 = -X22 T are split transposed; nothing above the diagonal of X11
    // and X22 is read, their parts get zeros there).  n1 >= n2 and n1 is a multiple
    // of 128, so four parts of n1 x n1 floats hold any pair of operands of this level; deeper
    // levels reuse the same scratch once this level's product has consumed it (one stream).
    if (pl.k % 4 != 0) return fail(HI2_ERR_DRIVER, "inverse_factor: wide inputs need k to be a multiple of 4");
    const int64_t part = n1 * n1;
    float *ah = pl.split, *al = ah + part, *bh = al + part, *bl = bh + part;
    const int64_t l1 = n1, l2 = ceil_div(n2, (int64_t)32) * 32;  // leading dimensions for kk = n1, n2
    // W (in the X21 slot) = A21 X11^T
    if ((rc = launch_split_block(a21, ld, n2, n1, ah, al, l1, false, false, pl.stream)) != HI2_OK) return rc;
    if ((rc = launch_split_block(x11, ld, n1, n1, bh, bl, l1, false, true, pl.stream)) != HI2_OK) return rc;
    rc = launch_gemm_tc(n2, n1, n1, ah, al, bh, bl, l1, x21, ld, GT_KB_LE_J, pl.status, pl.stream);
    if (rc != HI2_OK) return rc;
    // A22 -= W W^T (lower tiles)
    if ((rc = launch_split_block(x21, ld, n2, n1, ah, al, l1, false, false, pl.stream)) != HI2_OK) return rc;
    rc = launch_gemm_tc(n2, n2, n1, ah, al, ah, al, l1, a22, ld, GT_LOWER_OUT | GT_NEGATE | GT_ADD, pl.status,
                        pl.stream);
    if (rc != HI2_OK) return rc;
    // T (in the A21 slot) = W X11
    if ((rc = launch_split_block(x11, ld, n1, n1, bh, bl, l1, true, true, pl.stream)) != HI2_OK) return rc;
    rc = launch_gemm_tc(n2, n1, n1, ah, al, bh, bl, l1, a21, ld, GT_KB_GE_J, pl.status, pl.stream);
    if (rc != HI2_OK) return rc;
    rc = factor(pl, off + n1, n2);
    if (rc != HI2_OK) return rc;
    // X21 = -X22 T
    if ((rc = launch_split_block(x22, ld, n2, n2, ah, al, l2, false, true, pl.stream)) != HI2_OK) return rc;
    if ((rc = launch_split_block(a21, ld, n2, n1, bh, bl, l2, true, false, pl.stream)) != HI2_OK) return rc;
    return launch_gemm_tc(n2, n1, n2, ah, al, bh, bl, l2, x21, ld, GT_KA_LE_I | GT_NEGATE, pl.status, pl.stream);
  }
  const int m = (int)n2, k1 = (int)n1;
  // W (in the X21 slot) = A21 X11^T
  const ProductJob w{a21, x11, x21, m, k1, k1, GEMM_KB_LE_J, 1, 0, 0};
  if ((rc = launch_products(w, nullptr, ld, pl.stream)) != HI2_OK) return rc;
  // A22 -= W W^T (lower tiles), and T (in the A21 slot) = W X11, in one launch
  const ProductJob schur{x21, x21, a22, m, m, k1, GEMM_LOWER_OUT, 1, 1, 0};
  const ProductJob t{x21, x11, a21, m, k1, k1, GEMM_KB_GE_J, 0, 0, 0};
  if ((rc = launch_products(schur, &t, ld, pl.stream)) != HI2_OK) return rc;
  rc = factor(pl, off + n1, n2);
  if (rc != HI2_OK) return rc;
  // X21 = -X22 T
  const ProductJob last{x22, a21, x21, m, k1, m, GEMM_KA_LE_I, 0, 0, 1};
  return launch_products(last, nullptr, ld, pl.stream);
}

}  // namespace
}  // namespace hi2

extern "C" size_t hi2_inverse_factor_workspace_bytes(int64_t k) {
  if (k <= 0) return 0;
  return ((size_t)k * (size_t)hi2::padded(k) * 2 + hi2::split_floats(k)) * sizeof(float) + 256;
}

extern "C" int hi2_inverse_factor(const float* hs, const float* lam, int64_t k, float* u,
                                  void* workspace, size_t workspace_bytes, int32_t* info,
                                  void* stream) {
  using namespace hi2;
  HI2_REQUIRE(k > 0, "inverse_factor: k must be positive");
  HI2_REQUIRE(hs && lam && u && info && workspace, "inverse_factor: null pointer");
  if (workspace_bytes < hi2_inverse_factor_workspace_bytes(k))
    return fail(HI2_ERR_WORKSPACE, "inverse_factor: workspace too small");
  HI2_REQUIRE(aligned16(workspace), "inverse_factor: workspace must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  {  // per device, so not cached: a process may drive several
    if (cudaFuncSetAttribute(base_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BASE_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(product_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P_SMEM) != cudaSuccess)
      return fail(HI2_ERR_LAUNCH, "inverse_factor: cannot reserve shared memory");
  }
  Plan pl;
  // layout: one status word (256 bytes), A, X, then the TF32 parts
  pl.status = static_cast<int*>(workspace);
  pl.a = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + 256);
  pl.ld = padded(k);
  pl.x = pl.a + k * pl.ld;
  pl.split = split_floats(k) ? pl.x + k * pl.ld : nullptr;
  pl.k = k, pl.info = info, pl.stream = s;
  ChainGraph chain(s, chain_length(k));  // the whole recursion
  auto enqueue = [&]() -> int {
    if (cudaMemsetAsync(pl.status, 0, 256, s) != cudaSuccess)
      return fail(HI2_ERR_LAUNCH, "inverse_factor: memset failed");
    const dim3 grid((unsigned)k, (unsigned)ceil_div(k, 1024));
    const bool vec = k % 4 == 0 && aligned16(hs) && aligned16(u);
    if (vec) reverse_damp_kernel<true><<<grid, 256, 0, s>>>(hs, lam, k, pl.ld, pl.a);
    else reverse_damp_kernel<false><<<grid, 256, 0, s>>>(hs, lam, k, pl.ld, pl.a);
    int rc = check_launch("inverse_factor reverse");
    if (rc != HI2_OK) return rc;
    rc = factor(pl, 0, k);
    if (rc != HI2_OK) return rc;
    if (pl.split != nullptr) merge_status_kernel<<<1, 1, 0, s>>>(pl.status, info);
    if (vec) reverse_store_kernel<true><<<grid, 256, 0, s>>>(pl.x, k, pl.ld, u);
    else reverse_store_kernel<false><<<grid, 256, 0, s>>>(pl.x, k, pl.ld, u);
    return check_launch("inverse_factor store");
  };
  return chain.finish(enqueue(), "inverse_factor");
}
