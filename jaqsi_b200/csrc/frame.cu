// Kernels of frame plans (frame.h): parameters, forward and adjoint passes,
// chain rule.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <string>

#include "frame_dev.cuh"
#include "jq_internal.h"
#include "kernels.cuh"

namespace jq {
namespace {

// Gate parameters: U = (phase) Z^z P(f1) [[1, -t], [t, 1]] P(f0) X^piv / norm with
// P(f) = diag(1, e^{i f}), |t| <= 1, |f| <= pi / 2.  A phase is three shears,
// (re, im) -> re - tan(f/2) im, im + sin(f) re, re - tan(f/2) im: five FMA lanes an
// amplitude and gate, against ten (complex64, packed) or eight (complex128) for
// the 2x2 product.  Rounded shears keep determinant 1; a rounded pair (cos f, sin
// f) has a modulus off by half an ulp, which favours one role in every amplitude
// alike and does not average out (24 qubits, 20 layers, complex64: 5e-5 of the Z
// values against 1e-6).  X^piv moves the stage's base address.  Z^z is pushed to
// the end of the circuit, where it commutes with every Z word: on its way it turns
// t into -t where the mask crosses its functional (`flip`).  norm is applied every
// fourth stage.
template <typename F> struct FlagsOf { using T = uint32_t; };
template <> struct FlagsOf<double> { using T = uint64_t; };
// A dense block's row of the block matrices; a diagonal block has the second half.
template <typename F> struct __align__(16) GateRow {
  F t, tau0, sig0, pad0;              // rotation; phase before it: tan(f/2), sin f
  F tau1, sig1;                       // phase after it
  typename FlagsOf<F>::T flags, pad1; // 1: piv, 2: flip
};
static_assert(sizeof(GateRow<float>) == 4 * sizeof(float2) && sizeof(GateRow<double>) == 4 * sizeof(double2),
              "one 2x2 block");
template <typename C> struct RealOf;
template <> struct RealOf<float2> { using T = float; };
template <> struct RealOf<double2> { using T = double; };
template <typename C> using Real = typename RealOf<C>::T;
template <typename C> __device__ __forceinline__ const GateRow<Real<C>>* gate_at(const C* bm, int off, bool diag) {
  return reinterpret_cast<const GateRow<Real<C>>*>(bm + off - (diag ? 2 : 0));
}
template <typename C> __device__ __forceinline__ uint32_t gate_flags(const C* bm, int off, bool diag) {
  return static_cast<uint32_t>(gate_at(bm, off, diag)->flags);
}

// Stage tables in shared memory.
template <typename F> struct __align__(16) StageTab {
  F g[4][4];     // t, first phase of the gates (zeros: none)
  F h[4][2];     // second phase
  F scale;       // product of 1 / norm over the stages k.. of k's group of four
  uint32_t piv;
};
template <typename C> using Tab = StageTab<Real<C>>;
__device__ __forceinline__ void load_gate(const StageTab<float>& tb, int q, float (&c)[5]) {
  const float4 g = *reinterpret_cast<const float4*>(tb.g[q]);
  const float2 h = *reinterpret_cast<const float2*>(tb.h[q]);
  c[0] = g.x; c[1] = g.y; c[2] = g.z; c[3] = h.x; c[4] = h.y;
}
__device__ __forceinline__ void load_gate(const StageTab<double>& tb, int q, double (&c)[5]) {
  const double2 g = *reinterpret_cast<const double2*>(tb.g[q]), h = *reinterpret_cast<const double2*>(tb.h[q]);
  c[0] = g.x; c[1] = g.y; c[2] = tb.g[q][2]; c[3] = h.x; c[4] = h.y;
}

__device__ __forceinline__ void rot_pair(double2& x, double2& y, double t) {
  const double2 a = x;
  x.x = fma(-t, y.x, a.x);
  x.y = fma(-t, y.y, a.y);
  y.x = fma(t, a.x, y.x);
  y.y = fma(t, a.y, y.y);
}
__device__ __forceinline__ void rot_pair(float2& x, float2& y, float t) {
  const float2 a = x;
  x = __ffma2_rn(make_float2(-t, -t), y, a);
  y = __ffma2_rn(make_float2(t, t), a, y);
}
// v <- e^{i f} v, tau = tan(f/2), sig = sin f
template <typename C> __device__ __forceinline__ void shear(C& v, Real<C> tau, Real<C> sig) {
  v.x = fma(-tau, v.y, v.x);
  v.y = fma(sig, v.x, v.y);
  v.x = fma(-tau, v.y, v.x);
}

// The gates of a stage on 16 slots (slot bit q: role of gate q), and their inverse.
template <typename C> __device__ __forceinline__ void stage_forward(C (&v)[16], const Tab<C>& tb) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    Real<C> c[5];
    load_gate(tb, q, c);
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (!(j >> q & 1)) {
        const int m = j | (1 << q);
        shear(v[m], c[1], c[2]);
        rot_pair(v[j], v[m], c[0]);
        shear(v[m], c[3], c[4]);
      }
  }
}
template <typename C> __device__ __forceinline__ void stage_adjoint(C (&v)[16], const Tab<C>& tb) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    Real<C> c[5];
    load_gate(tb, q, c);
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (!(j >> q & 1)) {
        const int m = j | (1 << q);
        shear(v[m], -c[3], -c[4]);
        rot_pair(v[j], v[m], -c[0]);
        shear(v[m], -c[1], -c[2]);
      }
  }
}
__device__ __forceinline__ void mul_all(float2 (&v)[16], float f) {
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __fmul2_rn(v[j], make_float2(f, f));
}
__device__ __forceinline__ void mul_all(double2 (&v)[16], double f) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    v[j].x *= f;
    v[j].y *= f;
  }
}

// Shared-memory plan of a pass, in bytes.
template <typename C>
__host__ __device__ constexpr size_t tab_bytes(int nst) { return static_cast<size_t>(nst) * sizeof(Tab<C>); }
// Stage tables of one instance.
template <typename C, int LT>
__device__ __forceinline__ void pass_tables(const FrameStage* __restrict__ st, int nst, const C* __restrict__ bm, Tab<C>* tab) {
  using F = Real<C>;
  for (int i = threadIdx.x; i < nst * 8; i += 1 << LT) {
    const FrameStage& s = st[i >> 3];
    const int j = i & 7;
    Tab<C>& tb = tab[i >> 3];
    if (j < 4) {
      F c[5] = {0, 0, 0, 0, 0};
      if (j < s.ng) {
        const bool diag = s.diag >> (2 * j) & 1;
        const GateRow<F>* m = gate_at(bm, s.off[j], diag);
        if (!diag) { c[0] = m->t; c[1] = m->tau0; c[2] = m->sig0; }
        c[3] = m->tau1;
        c[4] = m->sig1;
      }
      tb.g[j][0] = c[0];
      tb.g[j][1] = c[1];
      tb.g[j][2] = c[2];
      tb.h[j][0] = c[3];
      tb.h[j][1] = c[4];
    } else if (j == 4) {
      uint32_t piv = 0;
      for (int q = 0; q < s.ng; ++q) piv |= (gate_flags(bm, s.off[q], s.diag >> (2 * q) & 1) & 1u) << q;
      tb.piv = piv;
    } else if (j == 5) {
      double f = 1.0;
      const int k = i >> 3, k1 = min(nst, (k | 3) + 1);
      for (int x = k; x < k1; ++x)
        for (int q = 0; q < st[x].ng; ++q)
          if (!(st[x].diag >> (2 * q) & 1)) {
            const double t = gate_at(bm, st[x].off[q], false)->t;  // the rounded one: exactly its norm
            f *= 1.0 + t * t;
          }
      tb.scale = static_cast<F>(1.0 / sqrt(f));
    }
  }
}

// One forward pass.  A tile (a coset of V) streams into shared memory while
// the previous one is computed; each stage loads its 16 slots a thread, applies
// up to four gates and stores.
//
// Bound by instruction issue and its latencies (57% of issue slots, 89 instructions
// an amplitude and pass of 12 gates; FMA pipe 43%, HBM 42% busy).  24 qubits, 20
// layers, complex64: 40 passes of 75 us for 133 stages against 66 passes of 60 us
// for 157, 4.19 -> 3.06 ms a call (tiles copied 8 bytes at a time instead of 16 cost
// 0.27 ms).  Five CTAs an SM; six (79 registers) were 18% slower.  Pairs of
// amplitudes in packed FMAs throughout: 1.5 times slower, register moves for every
// packed operand.
template <typename C, int T, int MINB>
__global__ void __launch_bounds__(1 << (T - 4), MINB)
    k_frame_fwd(C* __restrict__ state, const PassArg P, const FrameStage* __restrict__ stages,
                const C* __restrict__ bmat, int64_t bstride, int batch, int rev, int zero) {
  constexpr int LT = T - 4, NT = 1 << LT;
  constexpr uint32_t TB = sizeof(C) << T;     // bytes of a tile
  const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  Tab<C>* tab = reinterpret_cast<Tab<C>*>(smem + 2 * TB);
  uint32_t* soff = reinterpret_cast<uint32_t*>(tab + P.nst);
  uint16_t* tbs = reinterpret_cast<uint16_t*>(soff + 16 * P.nst);
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  asm volatile("griddepcontrol.launch_dependents;");
  const FrameStage* st = stages + P.st0;
  const int nst = P.nst;
  pass_setup<LT>(st, nst, tbs, soff);
  const uint32_t opos_lane = P.opos[lane];
  const uint32_t r_lane = (lane >> 2) < static_cast<uint32_t>(nst) ? st[lane >> 2].r[lane & 3] : 0u;
  const uint32_t s_lane = (lane >> 2) < static_cast<uint32_t>(nst) ? (st[lane >> 2].sbits >> (lane & 3) & 1u) : 0u;
  uint32_t gout = 0;  // this thread's part of the last stage's indices
#pragma unroll
  for (int i = 0; i < LT; ++i)
    if (tid >> i & 1u) gout ^= st[nst - 1].gtv[i];
  const TileCopy<C, LT> copy(P);
  const uint64_t tiles_per = 1ULL << P.nouter;
  const int64_t ntiles = static_cast<int64_t>(tiles_per) * batch;
  const uint64_t rmask = rev ? tiles_per - 1 : 0;
  auto load = [&](uint32_t dst, int64_t tl) {
    const uint32_t rep = tile_rep((static_cast<uint64_t>(tl) & (tiles_per - 1)) ^ rmask, opos_lane, P.nouter);
    if (zero) {  // the first pass of a run from |0..0>: nothing to read (24 qubits 3.09 -> 3.06 ms)
      copy.each(P, rep, dst, [&](uint32_t a, uint32_t b) {
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (a == 0) (sizeof(C) == 8 ? v.x : v.y) = sizeof(C) == 8 ? 0x3f800000u : 0x3ff00000u;  // 1
        *reinterpret_cast<uint4*>(smem + b) = v;
      });
      return;
    }
    const C* src = state + ((tl >> P.nouter) << P.nb);
    copy.each(P, rep, dst, [&](uint32_t a, uint32_t b) { cp_async16(sbase + b, src + a); });
  };
  // The first pass is launched in plain stream order, after the gate matrices were
  // written; a later one starts after the first has begun.  So the tables of the
  // first tile need no wait, only the states do: 20 qubits, forward + adjoint, 108
  // passes each way: 3.26 -> 3.09 ms with the adjoint passes launched ahead as
  // well, 2.70 ms with the tables formed before the wait; 24 qubits, 40 forward
  // passes: 3.20 -> 3.09 ms.
  int64_t last = -1;
  if (blockIdx.x < ntiles) {
    last = static_cast<int64_t>(blockIdx.x) >> P.nouter;
    pass_tables<C, LT>(st, nst, bmat + last * bstride, tab);
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (blockIdx.x < ntiles) load(0, blockIdx.x);
  cp_commit();
  uint32_t s = 0;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    if (tile + gridDim.x < ntiles) load(s ^ TB, tile + gridDim.x);
    cp_commit();
    const int64_t inst = tile >> P.nouter;
    const uint32_t rep = tile_rep((static_cast<uint64_t>(tile) & (tiles_per - 1)) ^ rmask, opos_lane, P.nouter);
    // bit 4 k + q: gate q of stage k has its roles exchanged in this tile
    const uint32_t flips = __ballot_sync(0xffffffffu, ((__popc(rep & r_lane) & 1u) ^ s_lane) != 0u);
    if (inst != last) {
      pass_tables<C, LT>(st, nst, bmat + inst * bstride, tab);
      last = inst;
    }
    cp_wait<1>();
    __syncthreads();
    C* g = state + (inst << P.nb);
    for (int k = 0; k < nst; ++k) {
      const Tab<C>& tb = tab[k];
      const uint32_t nib = k < kFrameBallot ? (flips >> (4 * k)) & 15u : st[k].sbits;
      const uint32_t* so = soff + 16 * k;
      const uint32_t e[4] = {so[1], so[2], so[4], so[8]};
      const uint32_t base = s ^ (static_cast<uint32_t>(tbs[k * NT + tid]) << 2);
      uint32_t a[16];
      C v[16];
      slot_offsets(e, base ^ so[nib ^ tb.piv], a);
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = lds<C>(a[j]);
      // group scale: the table entry of the group's first stage
      const bool rescale = (k & 3) == 3 || k + 1 == nst;
      stage_forward<C>(v, tb);
      if (rescale) mul_all(v, tab[k & ~3].scale);
      if (P.direct && k + 1 == nst) {
        const uint32_t ge[4] = {st[k].ge[0], st[k].ge[1], st[k].ge[2], st[k].ge[3]};
        slot_offsets(ge, rep ^ gout ^ slot_xor(ge, nib), a);
#pragma unroll
        for (int j = 0; j < 16; ++j) __stcs(g + a[j], v[j]);
      } else {
        slot_offsets(e, base ^ so[nib], a);
#pragma unroll
        for (int j = 0; j < 16; ++j) sts(a[j], v[j]);
        __syncthreads();
      }
    }
    if (!P.direct) {
      copy.each(P, rep, s, [&](uint32_t a, uint32_t b) { __stcs(reinterpret_cast<float4*>(g + a), lds<float4>(b)); });
    }
    __syncthreads();
    s ^= TB;
  }
}

// One adjoint pass: the pass's stages in reverse on psi and lambda, and the three
// components Im tr(sigma_k lam psi^dagger) of each gate's cotangent, all four
// gates of a stage at one point: a gate's reduced matrix does not depend on the
// other gates of its stage, and the generators of a rotation see only these
// three of its eight numbers.  A thread's and a warp's sums are of type A, tiles and
// warps add up in float64.  20 qubits, 50 layers, complex64 (forward +
// adjoint): 4.76 -> 2.60 ms a call; 16 qubits, 9 layers, complex128, three sets:
// 0.93 -> 0.43 ms.
template <typename C, typename A, int T, int MINB>
__global__ void __launch_bounds__(1 << (T - 4), MINB)
    k_frame_adj(const C* psi_in, C* psi, C* __restrict__ lam, const PassArg P, const FrameStage* __restrict__ stages,
                const C* __restrict__ bmat, int64_t bstride, double* __restrict__ gacc, int64_t gstride, int batch) {
  constexpr int LT = T - 4, NT = 1 << LT, NW = NT >= 32 ? NT / 32 : 1;
  using F = decltype(C::x);
  constexpr uint32_t TB = sizeof(C) << T;
  const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  asm volatile("griddepcontrol.launch_dependents;");
  Tab<C>* tab = reinterpret_cast<Tab<C>*>(smem + 2 * TB);
  uint32_t* soff = reinterpret_cast<uint32_t*>(tab + P.nst);
  uint16_t* tbs = reinterpret_cast<uint16_t*>(soff + 16 * P.nst);
  double* sacc = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(tbs) + tb_bytes(P.nst, NT));
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const FrameStage* st = stages + P.st0;
  const int nst = P.nst;
  pass_setup<LT>(st, nst, tbs, soff);
  for (int i = tid; i < NW * nst * 16; i += NT) sacc[i] = 0.0;
  const uint32_t opos_lane = P.opos[lane];
  const uint32_t r_lane = (lane >> 2) < static_cast<uint32_t>(nst) ? st[lane >> 2].r[lane & 3] : 0u;
  const uint32_t s_lane = (lane >> 2) < static_cast<uint32_t>(nst) ? (st[lane >> 2].sbits >> (lane & 3) & 1u) : 0u;
  uint32_t gout = 0;
#pragma unroll
  for (int i = 0; i < LT; ++i)
    if (tid >> i & 1u) gout ^= st[0].gtv[i];
  const TileCopy<C, LT> copy(P);
  const uint64_t tiles_per = 1ULL << P.nouter;
  const int64_t ntiles = static_cast<int64_t>(tiles_per) * batch;
  int64_t last = -1;
  if (blockIdx.x < ntiles) {  // before the wait: see k_frame_fwd
    last = static_cast<int64_t>(blockIdx.x) >> P.nouter;
    pass_tables<C, LT>(st, nst, bmat + last * bstride, tab);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  auto flush = [&](int64_t inst) {
    if (!gacc) return;
    for (int i = tid; i < nst * 12; i += NT) {
      const int k = i / 12, v = i - 12 * k, gt = st[k].gate[v / 3];
      if (gt < 0) continue;
      double x = 0.0;
      for (int w = 0; w < NW; ++w) x += sacc[(w * nst + k) * 16 + v];
      atomicAdd(&gacc[inst * gstride + 3 * gt + v % 3], x);
    }
  };
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t inst = tile >> P.nouter;
    const uint32_t rep = tile_rep(static_cast<uint64_t>(tile) & (tiles_per - 1), opos_lane, P.nouter);
    const uint32_t flips = __ballot_sync(0xffffffffu, ((__popc(rep & r_lane) & 1u) ^ s_lane) != 0u);
    const int64_t ibase = inst << P.nb;
    __syncthreads();
    copy.each(P, rep, 0, [&](uint32_t a, uint32_t b) {
      cp_async16(sbase + b, psi_in + ibase + a);
      cp_async16(sbase + (b ^ TB), lam + ibase + a);
    });
    cp_commit();
    if (inst != last) {
      if (last >= 0) {
        flush(last);
        __syncthreads();
        for (int i = tid; i < NW * nst * 16; i += NT) sacc[i] = 0.0;
      }
      pass_tables<C, LT>(st, nst, bmat + inst * bstride, tab);
      last = inst;
    }
    cp_wait<0>();
    __syncthreads();
    for (int k = nst - 1; k >= 0; --k) {
      const Tab<C>& tb = tab[k];
      const uint32_t nib = k < kFrameBallot ? (flips >> (4 * k)) & 15u : st[k].sbits;
      const uint32_t base = static_cast<uint32_t>(tbs[k * NT + tid]) << 2;
      const uint32_t* so = soff + 16 * k;
      const uint32_t e[4] = {so[1], so[2], so[4], so[8]};
      C p[16], l[16];
      {
        uint32_t a[16];
        slot_offsets(e, base ^ so[nib], a);
#pragma unroll
        for (int j = 0; j < 16; ++j) p[j] = lds<C>(a[j]);
        stage_adjoint<C>(p, tb);
#pragma unroll
        for (int j = 0; j < 16; ++j) l[j] = lds<C>(a[j] ^ TB);
        stage_adjoint<C>(l, tb);
      }
      F cs = tb.scale;  // norm of psi and lambda so far in this group
      if ((k & 3) == 0) {
        mul_all(p, cs);
        mul_all(l, cs);
        cs = F(1);
      }
      if (P.direct && k == 0) {
        uint32_t a[16];
        const uint32_t ge[4] = {st[0].ge[0], st[0].ge[1], st[0].ge[2], st[0].ge[3]};
        slot_offsets(ge, rep ^ gout ^ slot_xor(ge, nib ^ tb.piv), a);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          __stcs(psi + ibase + a[j], p[j]);
          __stcs(lam + ibase + a[j], l[j]);
        }
      } else {
        uint32_t a[16];
        slot_offsets(e, base ^ so[nib ^ tb.piv], a);
#pragma unroll
        for (int j = 0; j < 16; ++j) { sts(a[j], p[j]); sts(a[j] ^ TB, l[j]); }
      }
      if (gacc) {
        // -<lam|sigma|psi> imaginary parts: x, y, z of gates 0..3
        A v[16], w[16], lx[16], ly[16], px[16], py[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          lx[j] = l[j].x; ly[j] = l[j].y;
          px[j] = p[j].x; py[j] = p[j].y;
          w[j] = fma(ly[j], px[j], -(lx[j] * py[j]));
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          A x0 = 0, x1 = 0, y0 = 0, y1 = 0, z = 0;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (!(j >> q & 1)) {
              const int m = j | (1 << q);
              // Im(l0* p1) + Im(l1* p0), Re(l0* p1) - Re(l1* p0)
              x0 = fma(ly[j], px[m], x0);
              x1 = fma(lx[j], py[m], x1);
              x0 = fma(ly[m], px[j], x0);
              x1 = fma(lx[m], py[j], x1);
              y0 = fma(lx[j], px[m], y0);
              y1 = fma(lx[m], px[j], y1);
              y0 = fma(ly[j], py[m], y0);
              y1 = fma(ly[m], py[j], y1);
              z += w[j] - w[m];
            }
          v[3 * q] = x0 - x1;
          v[3 * q + 1] = y0 - y1;
          v[3 * q + 2] = z;
        }
        v[12] = v[13] = v[14] = v[15] = 0;
        const A x = warp_rs16(v, lane);
        if (!(lane & 1u)) sacc[(warp * nst + k) * 16 + (lane >> 1)] += static_cast<double>(x) * (static_cast<double>(cs) * cs);
      }
      if (!(P.direct && k == 0)) __syncthreads();
    }
    if (!P.direct) {
      copy.each(P, rep, 0, [&](uint32_t a, uint32_t b) {
        __stcs(reinterpret_cast<float4*>(psi + ibase + a), lds<float4>(b));
        __stcs(reinterpret_cast<float4*>(lam + ibase + a), lds<float4>(b ^ TB));
      });
    }
  }
  __syncthreads();
  if (last >= 0) flush(last);
}

// ---- parameters and chain rule ----------------------------------------------
// float64 2x2 product of a one-wire block's prims
__device__ void block_matrix(const DevBlock& blk, const DevPrim* prims, const DevOp* ops, const double* ang,
                             const double2* cpool, double2* acc) {
  double2 pm[4], tmp[4];
  prim_matrix(prims[blk.prim_begin], ops, ang, nullptr, cpool, acc, -1, tmp);
  for (int p = blk.prim_begin + 1; p < blk.prim_end; ++p) {
    prim_matrix(prims[p], ops, ang, nullptr, cpool, pm, -1, tmp);
    m_mul(pm, acc, tmp, 2);
    m_copy(tmp, acc, 2);
  }
}

// tan(f/2), sin f of w / |w| = e^{i f} for Re w >= 0, of -w otherwise (returns 1)
template <typename F> __device__ uint32_t put_phase(double2 w, F* tau, F* sig) {
  const double s = w.x < 0.0 ? -1.0 : 1.0, m = sqrt(w.x * w.x + w.y * w.y);
  *tau = static_cast<F>(s * w.y / (m + s * w.x));
  *sig = static_cast<F>(s * w.y / m);
  return w.x < 0.0;
}
// Parameters of a gate; returns its Z flag.
template <typename C> __device__ uint32_t put_gate(const double2* u, bool diag, C* out) {
  using F = Real<C>;
  GateRow<F>* o = reinterpret_cast<GateRow<F>*>(out - (diag ? 2 : 0));
  double2 a = u[0], b = u[1], c = u[2], d = u[3];
  uint32_t flags = 0, z = 0;
  if (diag) {
    z = put_phase(cmulc(d, a), &o->tau1, &o->sig1);
  } else {
    if (b.x * b.x + b.y * b.y > a.x * a.x + a.y * a.y) {
      a = u[1]; b = u[0]; c = u[3]; d = u[2];
      flags = 1;
    }
    // c / a = t e^{i f1}, d / a = e^{i (f0 + f1)}
    const double2 w1 = cmulc(c, a), w = cmulc(d, a);
    const double a2 = a.x * a.x + a.y * a.y, mc = sqrt(w1.x * w1.x + w1.y * w1.y);
    const double2 e1 = mc > 0.0 ? make_double2(w1.x / mc, w1.y / mc) : make_double2(1.0, 0.0);
    const uint32_t z0 = put_phase(cmulc(w, e1), &o->tau0, &o->sig0);
    z = z0 ^ put_phase(e1, &o->tau1, &o->sig1);
    const F t = static_cast<F>(mc / a2);
    o->t = z0 ? -t : t;
  }
  o->flags = flags;
  return z;
}
template <typename C> __device__ __forceinline__ void put_flip(C* out, bool diag) {
  GateRow<Real<C>>* o = reinterpret_cast<GateRow<Real<C>>*>(out - (diag ? 2 : 0));
  o->flags |= 2u;
  if (!diag) o->t = -o->t;
}

// Gate parameters of one instance a CTA, in schedule order; then the prefix
// XOR of the Z flags' functionals decides each gate's flip.
constexpr int kPrepThreads = 256;
template <typename C>
__global__ void __launch_bounds__(kPrepThreads)
    k_frame_prep(const FrameGate* __restrict__ gates, int ngates, const DevBlock* __restrict__ blocks,
                 const DevPrim* __restrict__ prims, const DevOp* __restrict__ ops, const double* __restrict__ angles,
                 int n_angles, const double2* __restrict__ cpool, C* __restrict__ bmat, int64_t bstride, ZeroFill z) {
  __shared__ uint32_t wsum[kPrepThreads / 32];
  const int64_t inst = blockIdx.x;
  const double* ang = angles ? angles + inst * n_angles : nullptr;
  C* bm = bmat + inst * bstride;
#pragma unroll
  for (int k = 0; k < 2; ++k)
    for (int64_t i = inst * kPrepThreads + threadIdx.x; i < z.n[k]; i += static_cast<int64_t>(gridDim.x) * kPrepThreads)
      z.p[k][i] = 0.0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (int g0 = 0; g0 < ngates; g0 += kPrepThreads) {
    const int g = g0 + threadIdx.x;
    FrameGate fg = {};
    uint32_t x = 0;
    if (g < ngates) {
      fg = gates[g];
      double2 u[4];
      block_matrix(blocks[fg.block], prims, ops, ang, cpool, u);
      if (put_gate(u, fg.diag, bm + fg.mat_off)) x = fg.r;
    }
    {
      uint32_t s = x;  // inclusive prefix XOR
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s ^= y;
      }
      if (lane == 31) wsum[warp] = s;
      __syncthreads();
      uint32_t before = carry, all = carry;
      for (int w = 0; w < kPrepThreads / 32; ++w) {
        if (w < warp) before ^= wsum[w];
        all ^= wsum[w];
      }
      before ^= s ^ x;
      if (g < ngates && (__popc(before & fg.m) & 1)) put_flip(bm + fg.mat_off, fg.diag);
      carry = all;
      __syncthreads();
    }
  }
}

// Rotation vector h of a prim (U^dagger dU = sum_k i h_k sigma_k per unit
// angle) and its action on a cotangent vector alpha_k = Im tr(sigma_k A):
// alpha of B A B^dagger.  Float64.
__device__ void rotate_axis(double* al, int axis, double th) {
  // B = exp(-i th/2 sigma_axis): rotates the vector by th about the axis
  double s, c;
  sincos(th, &s, &c);
  const int i = (axis + 1) % 3, j = (axis + 2) % 3;
  const double x = al[i], y = al[j];
  al[i] = c * x - s * y;
  al[j] = s * x + c * y;
}
__device__ void rotate_matrix(double* al, const double2* B) {
  // R_kl = Re tr(sigma_k B sigma_l B^dagger) / 2
  double r[3];
  for (int k = 0; k < 3; ++k) r[k] = 0.0;
  for (int l = 0; l < 3; ++l) {
    double2 S[4];
    m_zero(S, 2);
    if (l == 0) { S[1].x = 1; S[2].x = 1; }
    else if (l == 1) { S[1].y = -1; S[2].y = 1; }
    else { S[0].x = 1; S[3].x = -1; }
    double2 t[4], m[4];
    m_mul(B, S, t, 2);
    m_mul_bh(t, B, m, 2);
    r[0] += 0.5 * (m[1].x + m[2].x) * al[l];
    r[1] += 0.5 * (m[2].y - m[1].y) * al[l];  // tr(Y m) = -i m10 + i m01 -> real part m10.y - m01.y
    r[2] += 0.5 * (m[0].x - m[3].x) * al[l];
  }
  for (int k = 0; k < 3; ++k) al[k] = r[k];
}

template <typename C>
__global__ void k_frame_chain(const FrameGate* __restrict__ gates, int ngates, const DevBlock* __restrict__ blocks,
                              const DevPrim* __restrict__ prims, const DevOp* __restrict__ ops,
                              const double* __restrict__ angles, int n_angles, const double2* __restrict__ cpool,
                              const C* __restrict__ bmat, int64_t bstride, const double* __restrict__ gacc,
                              int64_t gstride, int batch, double* __restrict__ grad) {
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<int64_t>(batch) * ngates) return;
  const int64_t inst = idx / ngates;
  const int gi = static_cast<int>(idx - inst * ngates);
  const FrameGate fg = gates[gi];
  if (fg.grad < 0) return;
  const DevBlock blk = blocks[fg.block];
  const double* ang = angles + inst * n_angles;
  const double* acc = gacc + inst * gstride + 3 * fg.grad;
  double al[3] = {acc[0], acc[1], acc[2]};
  // cotangent of the pivoted block: X A X flips y and z (the sums are taken
  // after the block's diagonal and rotation parts, before X)
  const uint32_t fl = gate_flags(bmat + inst * bstride, fg.mat_off, fg.diag);
  if (fl & 1u) { al[1] = -al[1]; al[2] = -al[2]; }
  if (fl & 2u) { al[0] = -al[0]; al[1] = -al[1]; }  // conjugated by the Z pushed past it
  double* out = grad + inst * n_angles;
  for (int p = blk.prim_begin; p < blk.prim_end; ++p) {
    const DevPrim pr = prims[p];
    if (pr.form == PF_CONST || pr.op < 0) {
      double2 B[4], tmp[4];
      prim_matrix(pr, ops, ang, nullptr, cpool, B, -1, tmp);
      rotate_matrix(al, B);
      continue;
    }
    const DevOp op = ops[pr.op];
    const int naxes = op.kind == JQ_K_ROT ? 3 : 1;
    for (int j = 0; j < naxes; ++j) {
      int axis;
      if (op.kind == JQ_K_ROT) axis = j == 1 ? 1 : 2;
      else if (op.kind == JQ_K_PAULIROT) axis = op.px ? (op.pz ? 1 : 0) : 2;
      else axis = op.kind - JQ_K_RX;
      if (op.grad) atomicAdd(&out[op.angle_slot + j], -0.5 * al[axis]);
      rotate_axis(al, axis, ang[op.angle_slot + j]);
    }
  }
}

// ---- launches ------------------------------------------------------------------
template <typename C, int T> constexpr int fwd_minb() {
  // 128 threads (11 bits): complex64 5 CTAs an SM (100 registers), complex128 3 (168)
  return sizeof(C) == 8 ? (T >= 12 ? 2 : T == 11 ? 5 : 8) : (T >= 12 ? 1 : T == 11 ? 3 : 6);
}
template <typename C, typename A, int T> constexpr int adj_minb() {
  if (sizeof(A) < sizeof(double)) return T == 11 ? 4 : 0;
  return T >= 12 ? 1 : T == 11 ? 2 : sizeof(C) == 16 || T == 10 ? 4 : 8;
}

int pass_threads(const FramePass& p) { return 1 << (p.t - 4); }
template <typename C> size_t fwd_smem(const FramePass& p) {
  return (static_cast<size_t>(2) << p.t) * sizeof(C) + tab_bytes<C>(p.nst) + soff_bytes(p.nst) + tb_bytes(p.nst, pass_threads(p));
}
template <typename C> size_t adj_smem(const FramePass& p) {
  const int nt = pass_threads(p), nw = nt >= 32 ? nt / 32 : 1;
  return (static_cast<size_t>(2) << p.t) * sizeof(C) + tab_bytes<C>(p.nst) + soff_bytes(p.nst) + tb_bytes(p.nst, nt) +
         static_cast<size_t>(nw) * p.nst * 16 * sizeof(double);
}

template <typename C> const void* fwd_kernel(const FramePass& p) {
  switch (p.t) {
    case 9: return reinterpret_cast<const void*>(&k_frame_fwd<C, 9, fwd_minb<C, 9>()>);
    case 10: return reinterpret_cast<const void*>(&k_frame_fwd<C, 10, fwd_minb<C, 10>()>);
    case 11: return reinterpret_cast<const void*>(&k_frame_fwd<C, 11, fwd_minb<C, 11>()>);
    default: return reinterpret_cast<const void*>(&k_frame_fwd<C, 12, fwd_minb<C, 12>()>);
  }
}
// Cotangent sums of states below 2^16 amplitudes are float64 from the product on,
// as in the general reverse pass of that size; larger states sum in the run
// precision, as the specialised passes do.  (complex64, 11 bits: 224 registers and
// 2 CTAs an SM against 123 and 4; forward + adjoint, float32 -> float64 sums: 4 layers of
// 12 qubits 84.7 -> 92.9 us, 10 layers x 256 sets 238 -> 303, 20 layers of 15 qubits x
// 32 sets 666 -> 844, bound by the FP64 pipe and conversions: 3 CTAs an SM, 168
// registers, 870.  The general passes took 4.5 and 11.6 ms for these batches.)
template <typename C, typename A, int T> const void* adj_of() {
  return reinterpret_cast<const void*>(&k_frame_adj<C, A, T, adj_minb<C, A, T>()>);
}
template <typename C> const void* adj_kernel(const FramePass& p, int nb) {
  switch (p.t) {
    case 9: return adj_of<C, double, 9>();
    case 10: return adj_of<C, double, 10>();
    case 11: return nb < 16 ? adj_of<C, double, 11>() : adj_of<C, Real<C>, 11>();
    default: return adj_of<C, double, 12>();  // whole states only
  }
}

template <typename C> int upload_shapes(const FramePlan& fp, int nb, FrameDev* d) {
  for (const FramePass& p : fp.passes) {
    for (int adj = 0; adj < 2; ++adj) {
      const void* k = adj ? adj_kernel<C>(p, nb) : fwd_kernel<C>(p);
      const size_t smem = adj ? adj_smem<C>(p) : fwd_smem<C>(p);
      JQ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
      int n = 0;
      JQ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, pass_threads(p), smem));
      (adj ? d->adj_ctas : d->fwd_ctas).push_back(std::max(1, n));
    }
  }
  return JQ_OK;
}

template <typename C>
int forward_t(const jq_plan* plan, const FrameDev& d, C* state, int batch, const C* bmat, bool from_zero, int sm_count,
              cudaStream_t st) {
  const FramePlan& fp = plan->frame;
  const bool pdl = pdl_on(st);
  for (size_t i = 0; i < fp.passes.size(); ++i) {
    const FramePass& p = fp.passes[i];
    PassArg a = pass_arg(p, plan->n_bits, false);
    const int64_t ntiles = (1LL << p.nouter) * batch;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(std::min<int64_t>(ntiles, static_cast<int64_t>(sm_count) * d.fwd_ctas[i])));
    cfg.blockDim = dim3(static_cast<unsigned>(pass_threads(p)));
    cfg.dynamicSmemBytes = fwd_smem<C>(p);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl && i > 0 ? 1 : 0;
    const FrameStage* sp = d.stages;
    int64_t bs = plan->bmat_stride;
    int rev = static_cast<int>(i & 1), zero = from_zero && i == 0;
    void* args[] = {&state, &a, &sp, &bmat, &bs, &batch, &rev, &zero};
    JQ_CUDA(cudaLaunchKernelExC(&cfg, fwd_kernel<C>(p), args));
  }
  return JQ_OK;
}

template <typename C>
int adjoint_t(const jq_plan* plan, const FrameDev& d, const C* psi_in, C* psi, C* lam, int batch, const C* bmat,
              double* gacc, int64_t gstride, int sm_count, cudaStream_t st) {
  const FramePlan& fp = plan->frame;
  const bool pdl = pdl_on(st);
  for (size_t i = fp.passes.size(); i-- > 0;) {
    const FramePass& p = fp.passes[i];
    PassArg a = pass_arg(p, plan->n_bits, true);
    const int64_t ntiles = (1LL << p.nouter) * batch;
    const FrameStage* sp = d.stages;
    int64_t bs = plan->bmat_stride;
    const C* in = i + 1 == fp.passes.size() ? psi_in : psi;
    void* args[] = {&in, &psi, &lam, &a, &sp, &bmat, &bs, &gacc, &gstride, &batch};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(std::min<int64_t>(ntiles, static_cast<int64_t>(sm_count) * d.adj_ctas[i])));
    cfg.blockDim = dim3(static_cast<unsigned>(pass_threads(p)));
    cfg.dynamicSmemBytes = adj_smem<C>(p);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl && i + 1 < fp.passes.size() ? 1 : 0;
    JQ_CUDA(cudaLaunchKernelExC(&cfg, adj_kernel<C>(p, plan->n_bits), args));
  }
  return JQ_OK;
}

}  // namespace

int frame_tables(const FramePlan& fp, FrameDev* d) {
  const size_t ns = std::max<size_t>(1, fp.stages.size()), ng = std::max<size_t>(1, fp.gates.size());
  JQ_CUDA(cudaMalloc(reinterpret_cast<void**>(&d->stages), ns * sizeof(FrameStage)));
  JQ_CUDA(cudaMalloc(reinterpret_cast<void**>(&d->gates), ng * sizeof(FrameGate)));
  if (!fp.stages.empty())
    JQ_CUDA(cudaMemcpy(d->stages, fp.stages.data(), fp.stages.size() * sizeof(FrameStage), cudaMemcpyHostToDevice));
  if (!fp.gates.empty())
    JQ_CUDA(cudaMemcpy(d->gates, fp.gates.data(), fp.gates.size() * sizeof(FrameGate), cudaMemcpyHostToDevice));
  return JQ_OK;
}

int frame_upload(const jq_plan* plan, FrameDev* d) {
  const FramePlan& fp = plan->frame;
  if (!fp.on) return JQ_OK;
  const int rc = frame_tables(fp, d);
  if (rc) return rc;
  return plan->dtype == JQ_C64 ? upload_shapes<float2>(fp, plan->n_bits, d) : upload_shapes<double2>(fp, plan->n_bits, d);
}

void frame_free(FrameDev* d) {
  if (d->stages) cudaFree(d->stages);
  if (d->gates) cudaFree(d->gates);
  d->stages = nullptr;
  d->gates = nullptr;
}

int frame_prep(const jq_plan* plan, const FrameDev& d, const DevBlock* blocks, const DevPrim* prims, const DevOp* ops,
               const double* cpool, int batch, const double* angles, void* bmat, const ZeroFill& z, cudaStream_t st) {
  const int ng = static_cast<int>(plan->frame.gates.size());
  if (ng == 0 && z.n[0] + z.n[1] == 0) return JQ_OK;
  const double2* cp = reinterpret_cast<const double2*>(cpool);
  if (plan->dtype == JQ_C64)
    k_frame_prep<float2><<<batch, kPrepThreads, 0, st>>>(d.gates, ng, blocks, prims, ops, angles, plan->n_angles, cp,
                                                         static_cast<float2*>(bmat), plan->bmat_stride, z);
  else
    k_frame_prep<double2><<<batch, kPrepThreads, 0, st>>>(d.gates, ng, blocks, prims, ops, angles, plan->n_angles, cp,
                                                          static_cast<double2*>(bmat), plan->bmat_stride, z);
  JQ_CUDA(cudaGetLastError());
  return JQ_OK;
}

int frame_forward(const jq_plan* plan, const FrameDev& d, void* state, int batch, const void* bmat, bool from_zero,
                  int sm_count, cudaStream_t st) {
  return plan->dtype == JQ_C64
             ? forward_t<float2>(plan, d, static_cast<float2*>(state), batch, static_cast<const float2*>(bmat), from_zero,
                                 sm_count, st)
             : forward_t<double2>(plan, d, static_cast<double2*>(state), batch, static_cast<const double2*>(bmat), from_zero,
                                  sm_count, st);
}

int frame_adjoint(const jq_plan* plan, const FrameDev& d, const void* psi_in, void* psi, void* lam, int batch,
                  const void* bmat, double* gacc, int64_t gstride, int sm_count, cudaStream_t st) {
  return plan->dtype == JQ_C64
             ? adjoint_t<float2>(plan, d, static_cast<const float2*>(psi_in), static_cast<float2*>(psi),
                                 static_cast<float2*>(lam), batch, static_cast<const float2*>(bmat), gacc, gstride, sm_count, st)
             : adjoint_t<double2>(plan, d, static_cast<const double2*>(psi_in), static_cast<double2*>(psi),
                                  static_cast<double2*>(lam), batch, static_cast<const double2*>(bmat), gacc, gstride, sm_count, st);
}

int frame_chain(const jq_plan* plan, const FrameDev& d, const DevBlock* blocks, const DevPrim* prims, const DevOp* ops,
                const double* cpool, int batch, const double* angles, const void* bmat, const double* gacc,
                int64_t gstride, double* grad_angles, cudaStream_t st) {
  const int ng = static_cast<int>(plan->frame.gates.size());
  if (ng == 0 || !grad_angles) return JQ_OK;
  const int64_t work = static_cast<int64_t>(ng) * batch;
  const unsigned grid = static_cast<unsigned>((work + 63) / 64);
  const double2* cp = reinterpret_cast<const double2*>(cpool);
  if (plan->dtype == JQ_C64)
    k_frame_chain<float2><<<grid, 64, 0, st>>>(d.gates, ng, blocks, prims, ops, angles, plan->n_angles, cp,
                                               static_cast<const float2*>(bmat), plan->bmat_stride, gacc, gstride, batch,
                                               grad_angles);
  else
    k_frame_chain<double2><<<grid, 64, 0, st>>>(d.gates, ng, blocks, prims, ops, angles, plan->n_angles, cp,
                                                static_cast<const double2*>(bmat), plan->bmat_stride, gacc, gstride,
                                                batch, grad_angles);
  JQ_CUDA(cudaGetLastError());
  return JQ_OK;
}

}  // namespace jq
