// The last step of a second moment: the finished item tiles are added to S, upper triangle and mirror.
#pragma once

#include "common.cuh"

namespace hi2 {

constexpr int MR_SIDE = 64;  // divides the sides of every kernel's tiles
constexpr int MR_LD = MR_SIDE + 1;

// S[i][j] += sum over splits (ascending) of the item tiles, for i <= j; S[j][i] = S[i][j].  Tiles are TM x TN,
// row-major; Slot gives the place of the tile that holds row block i / TM, column block j / TN.
//
// A thread block takes a 64 x 64 piece on or above the diagonal and writes it twice, as it is and
// transposed through shared memory: all accesses are 16 bytes a lane along rows.  (Mirroring element by
// element scattered one sector per element.)  Bound by memory: 717 -> 169 us for the 1.0 GB of
// K = 11008 with one split, 23 -> 8 us at K = 2048 with two.
template <int TM, int TN, typename Slot>
__global__ void __launch_bounds__(256)
moment_reduce_kernel(const float* __restrict__ scratch, int splits, size_t split_stride, int64_t k, float* __restrict__ s,
                     const int* __restrict__ status, Slot slot) {
  static_assert(TM % MR_SIDE == 0 && TN % MR_SIDE == 0, "a piece lies in one tile");
  __shared__ float piece[MR_SIDE * MR_LD];
  // a product that gave up on a bounded wait left stale or partial tiles: S stays as it was and the
  // caller sees the status word
  if (*status != 0) return;
  const int64_t i0 = (int64_t)blockIdx.y * MR_SIDE, j0 = (int64_t)blockIdx.x * MR_SIDE;
  if (j0 < i0) return;
  const int q = (threadIdx.x & 15) * 4, r0 = threadIdx.x >> 4;  // columns q .. q + 3 of rows r0 + 16 a
  const float* tile = scratch + (size_t)slot((int)(i0 / TM), (int)(j0 / TN)) * ((size_t)TM * TN) +
                      (size_t)(i0 % TM) * TN + (size_t)(j0 % TN) + q;
  const bool cols = j0 + q < k;  // k is a multiple of 16
  float4 v[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) v[a] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int sp = 0; sp < splits; ++sp) {
    float4 t[4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
      t[a] = *reinterpret_cast<const float4*>(tile + (size_t)sp * split_stride + (size_t)(r0 + 16 * a) * TN);
#pragma unroll
    for (int a = 0; a < 4; ++a) v[a].x += t[a].x, v[a].y += t[a].y, v[a].z += t[a].z, v[a].w += t[a].w;
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = r0 + 16 * a;
    const bool in = cols && i0 + r < k;
    float4* at = reinterpret_cast<float4*>(s + (i0 + r) * k + j0 + q);
    if (in) {
      const float4 old = *at;
      v[a] = make_float4(old.x + v[a].x, old.y + v[a].y, old.z + v[a].z, old.w + v[a].w);
      if (i0 != j0) *at = v[a];
    }
    float* p = piece + r * MR_LD + q;
    p[0] = v[a].x, p[1] = v[a].y, p[2] = v[a].z, p[3] = v[a].w;
  }
  __syncthreads();
#pragma unroll
  for (int a = 0; a < 4; ++a) {  // row j0 + r of S, columns i0 + q ..
    const int r = r0 + 16 * a;
    if (j0 + r >= k || i0 + q >= k) continue;
    float o[4];
#pragma unroll
    for (int t = 0; t < 4; ++t)
      o[t] = (i0 == j0 && r <= q + t) ? piece[r * MR_LD + q + t] : piece[(q + t) * MR_LD + r];
    *reinterpret_cast<float4*>(s + (j0 + r) * k + i0 + q) = make_float4(o[0], o[1], o[2], o[3]);
  }
}

template <int TM, int TN, typename Slot>
int launch_moment_reduce(const float* scratch, int splits, int tiles, int64_t k, float* s, const int* status, Slot slot,
                         cudaStream_t stream, const char* what) {
  const unsigned side = (unsigned)ceil_div(k, MR_SIDE);
  moment_reduce_kernel<TM, TN, Slot><<<dim3(side, side), 256, 0, stream>>>(
      scratch, splits, (size_t)tiles * TM * TN, k, s, status, slot);
  return check_launch(what);
}

}  // namespace hi2
