// Shared definitions of the sm_100a kernels behind the C-ABI declared in include/hi2_b200.h.
//
// Arithmetic convention: the whole library is compiled with -fmad=false, so `a * b + c` is two
// roundings exactly as written (the reference path rounds every product and sum separately).
// Where a fused multiply-add is wanted it is spelled fmaf()/fma().
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/hi2_b200.h"

namespace hi2 {

void set_error(const char* fmt, ...);
void note_launch();  // one more kernel launch enqueued by this library (process-wide counter)

inline int fail(int code, const char* what) {
  set_error("%s", what);
  return code;
}

inline int check_launch(const char* what) {
  note_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("%s: %s", what, cudaGetErrorString(e));
    return HI2_ERR_LAUNCH;
  }
  return HI2_OK;
}

// A long chain of short kernels queued as ONE graph launch.  Between construction and finish()
// everything the calling thread launches on `stream` is captured instead of run; finish()
// instantiates the captured graph and launches it on the stream.  Why: a stream's launch queue
// holds about a thousand entries, so a chain of 1700 small kernels (the inverse factor of one
// input) throttles the host to the GPU's pace until it has drained, and the host cannot feed the
// other streams meanwhile - the chains of four inputs then run one after the other instead of
// side by side; as a graph the chain costs the host one launch and its kernels start back to back.
// A stream that is already being captured by the caller is left alone (the launches then join the
// caller's graph), and the legacy default stream, which cannot be captured, takes every chain plain.  So
// does any stream a chain of at most CHAIN_PLAIN launches: it fits the queue, and the GPU starts on it
// while a graph would still be captured and instantiated.  Measured on a stream of its own, graph / plain,
// ms: inverse factor K = 1024 (29 launches) 0.83 / 0.57, 3072 (103) 2.18 / 1.74, 4096 (155) 3.00 / 2.51;
// column loop 1024 x 6144 (95) 1.97 / 1.76, 1024 x 8192 (127) 2.66 / 2.42, 1024 x 11008 (171) 3.66 / 3.39.
// So a chain alone is quicker plain at every length, and the line is not where the two cross: it is a
// tenth of the queue, which is what several streams share.  A decoder layer with its chains side by side:
// all as graphs 54.0 ms, by the line 54.1, all plain 52.9; a layer of five experts 24.7, 21.5, 21.2 (runs
// of one kind differ by 2 to 4 %).  Finished graphs are destroyed on later calls, once their completion
// event has passed.
class ChainGraph {
 public:
  static constexpr int64_t CHAIN_PLAIN = 96;
  explicit ChainGraph(cudaStream_t stream, int64_t launches = INT64_MAX);
  // rc: the status of the launches issued since construction.  Returns rc if it is an error (the
  // captured work is dropped), else the status of instantiating and launching the graph.
  int finish(int rc, const char* what);
  ~ChainGraph();

 private:
  cudaStream_t stream_;
  bool capturing_ = false;
};

// Launch of a link of a chain of short kernels: the kernel may be set up while its predecessor in the
// stream still runs (programmatic dependent launch; in a captured chain the edge is a programmatic
// one).  Every such kernel calls chain_wait() before it touches global memory, which returns once the
// predecessor has finished and its writes are visible; since every link waits for the one before it,
// order along the stream is kept for whatever follows.  A predecessor calls chain_next() when all that
// is left to it is its stores: the successor's thread blocks hold their registers and shared memory
// while they wait, and set up any earlier they kept other streams' kernels off the SMs (a decoder layer
// with its tables and factor chains side by side 53.6 -> 58.6 ms).
template <typename... Params, typename... Args>
inline void launch_link(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = grid, config.blockDim = block, config.dynamicSmemBytes = smem, config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute, config.numAttrs = 1;
  cudaLaunchKernelEx(&config, kernel, Params(args)...);
}
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// One flag per 16-column group: an array on the device, or bits in the kernel's own arguments for a caller
// whose flags are on the host (they decide a few hundred bits; a copy to the device cost 25 us of host
// time per call).
struct GroupFlags {
  static constexpr int64_t MAX_GROUPS = 8192;
  const uint8_t* device;
  uint32_t bits[MAX_GROUPS / 32];

  static GroupFlags on_device(const uint8_t* flags) {
    GroupFlags f;
    f.device = flags;
    return f;
  }
  static GroupFlags on_host(const uint8_t* flags, int64_t groups) {
    GroupFlags f;
    f.device = nullptr;
    for (int64_t i = 0; i < MAX_GROUPS / 32; ++i) f.bits[i] = 0;
    for (int64_t g = 0; g < groups; ++g) f.bits[g >> 5] |= (flags[g] != 0 ? 1u : 0u) << (g & 31);
    return f;
  }
  __device__ __forceinline__ bool on(int64_t g) const {
    return device != nullptr ? __ldg(device + g) != 0 : ((bits[g >> 5] >> (g & 31)) & 1u) != 0;
  }
};

#define HI2_REQUIRE(cond, msg)                         \
  do {                                                 \
    if (!(cond)) return ::hi2::fail(HI2_ERR_ARG, msg); \
  } while (0)

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

__host__ __device__ inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// torch.clamp(lo, hi) semantics: NaN stays NaN.
__device__ __forceinline__ float clamp_keep_nan(float v, float lo, float hi) {
  v = (v < lo) ? lo : v;
  v = (v > hi) ? hi : v;
  return v;
}

__device__ __forceinline__ float round_f16(float v) { return __half2float(__float2half_rn(v)); }

// Division by a value that stays fixed over many quotients.  r is the correctly rounded
// reciprocal; `fast` is false when b is outside a comfortable normal range or its significand is
// all ones (the one case Markstein's correction step does not cover): then the IEEE division
// is used, so div_by returns exactly what __fdiv_rn would give.
struct Recip {
  float r;
  bool fast;
};
__device__ __forceinline__ Recip make_recip(float b) {
  const float ab = fabsf(b);
  Recip rc;
  rc.fast = ab > 1e-18f && ab < 1e18f && (__float_as_uint(b) & 0x7fffffu) != 0x7fffffu;
  rc.r = __frcp_rn(b);
  return rc;
}

// __fdiv_rn(a, b): q0 = a * r is a faithful quotient, one fused correction step makes it the
// correctly rounded one (Markstein).  a is assumed finite and not denormal-small.
__device__ __forceinline__ float div_by(float a, float b, Recip rc) {
  if (!rc.fast) return __fdiv_rn(a, b);
  const float q0 = a * rc.r;
  return fmaf(fmaf(-q0, b, a), rc.r, q0);
}

}  // namespace hi2
