// Device code shared by the frame plans' kernels (frame.h).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <string>

#include "frame.h"

namespace jq {
void set_error(const std::string& msg);

namespace {

#define JQ_CUDA(expr)                                                                       \
  do {                                                                                      \
    cudaError_t _e = (expr);                                                                \
    if (_e != cudaSuccess) {                                                                \
      set_error(std::string("CUDA error: ") + cudaGetErrorString(_e) + " at " #expr);       \
      return JQ_ECUDA;                                                                      \
    }                                                                                       \
  } while (0)

// Kernel argument of one pass.
struct PassArg {
  uint32_t g[kFrameMaxT];
  uint32_t cs[kFrameMaxT];
  uint32_t opos[32];
  int32_t nb, nouter;
  int32_t st0, nst;
  int32_t direct;
};

__device__ __forceinline__ void cp_async16(uint32_t sa, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Shared-memory accesses by byte offset; two tiles lie at offsets 0 and 2^T
// amplitudes, so that tile, thread and slot parts of an offset combine by XOR.
extern __shared__ __align__(16) unsigned char smem[];
template <typename C> __device__ __forceinline__ C lds(uint32_t a) { return *reinterpret_cast<const C*>(smem + a); }
template <typename C> __device__ __forceinline__ void sts(uint32_t a, C v) { *reinterpret_cast<C*>(smem + a) = v; }

// Offset of register slot j = XOR of the register vectors of its bits.
__device__ __forceinline__ void slot_offsets(const uint32_t (&e)[4], uint32_t base, uint32_t (&a)[16]) {
  a[0] = base;
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int j = 0; j < (1 << q); ++j) a[j | (1 << q)] = a[j] ^ e[q];
}
// The same over N vectors.
template <int N>
__device__ __forceinline__ void xor_offsets(const uint32_t* v, uint32_t base, uint32_t (&a)[1 << N]) {
  a[0] = base;
#pragma unroll
  for (int q = 0; q < N; ++q)
#pragma unroll
    for (int j = 0; j < (1 << q); ++j) a[j | (1 << q)] = a[j] ^ v[q];
}
// A tile's copy: chunks of 16 bytes, 2^CB values; a thread copies 2^(4-CB) of them.
template <typename E, int LT> struct TileCopy {
  static constexpr int CB = sizeof(E) == 4 ? 2 : sizeof(E) == 8 ? 1 : 0, N = 4 - CB;
  uint32_t gtid = 0, stid = 0;
  __device__ __forceinline__ explicit TileCopy(const PassArg& P) {
    const uint32_t tid = threadIdx.x;
#pragma unroll
    for (int i = 0; i < LT; ++i)
      if (tid >> i & 1u) {
        gtid ^= P.g[CB + i];
        stid ^= P.cs[CB + i];
      }
  }
  // f(index from the tile's instance, shared offset) of every chunk
  template <typename Fn> __device__ __forceinline__ void each(const PassArg& P, uint32_t rep, uint32_t s, Fn f) const {
    uint32_t a[1 << N], b[1 << N];
    xor_offsets<N>(P.g + CB + LT, rep ^ gtid, a);
    xor_offsets<N>(P.cs + CB + LT, s ^ stid, b);
#pragma unroll
    for (int i = 0; i < (1 << N); ++i) f(a[i], b[i]);
  }
};
__device__ __forceinline__ uint32_t slot_xor(const uint32_t* e, uint32_t n) {
  return ((n & 1u) ? e[0] : 0u) ^ ((n & 2u) ? e[1] : 0u) ^ ((n & 4u) ? e[2] : 0u) ^ ((n & 8u) ? e[3] : 0u);
}

__host__ __device__ constexpr size_t soff_bytes(int nst) { return static_cast<size_t>(nst) * 16 * sizeof(uint32_t); }
__host__ __device__ constexpr size_t tb_bytes(int nst, int threads) {
  return (static_cast<size_t>(nst) * threads * sizeof(uint16_t) + 15) & ~static_cast<size_t>(15);
}

// Tile-independent offsets of a pass: thread bases (in 4 bytes) and slots.
template <int LT>
__device__ __forceinline__ void pass_setup(const FrameStage* __restrict__ st, int nst, uint16_t* tbs, uint32_t* soff) {
  const uint32_t tid = threadIdx.x;
  for (int k = 0; k < nst; ++k) {
    uint32_t b = 0;
#pragma unroll
    for (int i = 0; i < LT; ++i)
      if (tid >> i & 1u) b ^= st[k].tv[i];
    tbs[k * (1 << LT) + tid] = static_cast<uint16_t>(b >> 2);
  }
  for (int i = tid; i < nst * 16; i += 1 << LT) soff[i] = slot_xor(st[i >> 4].e, i & 15);
}

// Representative of tile ti: its index bits at the free positions.
__device__ __forceinline__ uint32_t tile_rep(uint64_t ti, uint32_t opos_lane, int nouter) {
  const int lane = threadIdx.x & 31;
  const uint32_t v = (lane < nouter && (ti >> lane & 1ULL)) ? opos_lane : 0u;
  return __reduce_or_sync(0xffffffffu, v);
}

// Warp reduce-scatter of 16 per-lane sums by recursive halving (16 shuffles);
// even lane 2 v ends with the sum of value v.
template <typename F>
__device__ __forceinline__ F warp_rs16(F (&v)[16], unsigned lane) {
#pragma unroll
  for (int o = 16, n = 16; o > 1; o >>= 1, n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const F send = up ? v[i] : v[i + n / 2];
      const F keep = up ? v[i + n / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}


// programmatic stream serialisation of a pass: not while the stream is captured
bool pdl_on(cudaStream_t st) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
}

PassArg pass_arg(const FramePass& p, int nb, bool adjoint) {
  PassArg a;
  std::memset(&a, 0, sizeof(a));
  std::memcpy(a.g, p.g, sizeof(a.g));
  std::memcpy(a.cs, p.cs, sizeof(a.cs));
  std::memcpy(a.opos, p.opos, sizeof(a.opos));
  a.nb = nb;
  a.nouter = p.nouter;
  a.st0 = p.st0;
  a.nst = p.nst;
  a.direct = adjoint ? p.adirect : p.direct;
  return a;
}

}  // namespace
}  // namespace jq
