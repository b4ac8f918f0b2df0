// Noisy circuits in the Pauli basis (frame.h): expectation values of Pauli words
// on a density matrix and their gradients.
//
// rho = 2^-n sum_P r_P P with real r_P = tr(P rho): half the bytes of the matrix
// entries.  A one-qubit gate or channel (trace preserving) is a real 4x4 matrix
// with first row (1, 0, 0, 0): 12 FMA on four values, where its complex 4x4
// superoperator takes 64 on the (ket, bra) entries.  An expectation value is one
// coefficient, a seed of the reverse pass one nonzero.
//
// Index: wire w has x bit 2 (n-1-w) and z bit 2 (n-1-w) + 1; I, X, Z, Y = 0..3.  A
// linear permutation of the basis, |v> -> |A v>, maps X^x Z^z to X^{A x} Z^{A^-T z}
// without a sign, so what is stored is s_P = (-1)^floor(y/2) r_P, y the number of
// Y factors: the frame moves, the values stay.  Inside a stage the relative signs of its
// two wires' Y entries follow from the parity of y over the other wires, the
// quadratic form sum_w x_w z_w that every such permutation preserves.
#include <cuda_runtime.h>

#include <algorithm>

#include "frame_dev.cuh"
#include "jq_internal.h"
#include "kernels.cuh"

namespace jq {
namespace {

// Rows X, Z, Y of the transfer matrices of a stage's two wires.
template <typename F> struct __align__(16) PTab { F m[2][12]; };

__device__ __forceinline__ float flip_sign(float v, uint32_t s) { return __uint_as_float(__float_as_uint(v) ^ (s << 31)); }
__device__ __forceinline__ double flip_sign(double v, uint32_t s) {
  return __hiloint2double(__double2hiint(v) ^ static_cast<int>(s << 31), __double2loint(v));
}
// parity of the number of Y factors
__device__ __forceinline__ uint32_t y_parity(uint32_t g) { return __popc(g & (g >> 1) & 0x55555555u) & 1u; }

// Signs.  In a stage of two wires slot (a, b) = a + 4 b carries (-1)^(p [a = Y] + p
// [b = Y] + [a = Y][b = Y]), p the y parity of slot 0.  To a wire's matrix that
// is one sign on its entries with exactly one Y: (-1)^p, and the other one
// where the other wire is Y, so the five entries change sign (flip_odd) and the
// values need none: 10 instead of 28 sign operations on 16 values.
template <typename F> __device__ __forceinline__ void flip_odd(F (&c)[12], uint32_t p) {
  c[3] = flip_sign(c[3], p);
  c[7] = flip_sign(c[7], p);
  c[8] = flip_sign(c[8], p);
  c[9] = flip_sign(c[9], p);
  c[10] = flip_sign(c[10], p);
}
__device__ __host__ constexpr bool odd_entry(int e) { return e == 3 || (e >= 7 && e <= 10); }
// A stage of one wire: its register vectors 2 and 3 are not a wire's, and each of
// the four columns has its own parity.
template <typename F> __device__ __forceinline__ void column_signs(F (&v)[16], uint32_t g0, const FrameStage& st) {
  v[3] = flip_sign(v[3], y_parity(g0));
  v[7] = flip_sign(v[7], y_parity(g0 ^ st.ge[2]));
  v[11] = flip_sign(v[11], y_parity(g0 ^ st.ge[3]));
  v[15] = flip_sign(v[15], y_parity(g0 ^ st.ge[2] ^ st.ge[3]));
}

// The 12 entries of a wire's matrix, by 16-byte loads.
__device__ __forceinline__ void load12(const float* m, float (&c)[12]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float4 v = reinterpret_cast<const float4*>(m)[i];
    c[4 * i] = v.x; c[4 * i + 1] = v.y; c[4 * i + 2] = v.z; c[4 * i + 3] = v.w;
  }
}
__device__ __forceinline__ void load12(const double* m, double (&c)[12]) {
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    const double2 v = reinterpret_cast<const double2*>(m)[i];
    c[2 * i] = v.x; c[2 * i + 1] = v.y;
  }
}

// v <- M v on wire a (S = 1) or b (S = 4); PAIR: the other wire's Y (group 3)
// takes the odd entries with the other sign
template <int S, bool PAIR, typename F> __device__ __forceinline__ void apply_m(F (&v)[16], const F (&m)[12]) {
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    F c[12];
#pragma unroll
    for (int e = 0; e < 12; ++e) c[e] = PAIR && g == 3 && odd_entry(e) ? -m[e] : m[e];
    const int b = S == 1 ? 4 * g : g;
    const F a0 = v[b], a1 = v[b + S], a2 = v[b + 2 * S], a3 = v[b + 3 * S];
#pragma unroll
    for (int r = 0; r < 3; ++r)
      v[b + (r + 1) * S] = fma(c[4 * r + 3], a3, fma(c[4 * r + 2], a2, fma(c[4 * r + 1], a1, c[4 * r] * a0)));
  }
}
// v <- M^T v
template <int S, bool PAIR, typename F> __device__ __forceinline__ void apply_mt(F (&v)[16], const F (&m)[12]) {
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    F c[12];
#pragma unroll
    for (int e = 0; e < 12; ++e) c[e] = PAIR && g == 3 && odd_entry(e) ? -m[e] : m[e];
    const int b = S == 1 ? 4 * g : g;
    const F a1 = v[b + S], a2 = v[b + 2 * S], a3 = v[b + 3 * S];
    v[b] = fma(c[8], a3, fma(c[4], a2, fma(c[0], a1, v[b])));
#pragma unroll
    for (int r = 1; r < 4; ++r) v[b + r * S] = fma(c[8 + r], a3, fma(c[4 + r], a2, c[r] * a1));
  }
}
// g[4 (i - 1) + j] = sum of l (entry i of the wire) times x (entry j), i = 1..3
template <int S, bool PAIR, typename F, typename A>
__device__ __forceinline__ void outer_sum(const F (&l)[16], const F (&x)[16], A (&g)[16]) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      A a = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int b = S == 1 ? 4 * q : q;
        const A y = x[b + j * S];
        a = fma(static_cast<A>(l[b + (i + 1) * S]), PAIR && q == 3 && odd_entry(4 * i + j) ? -y : y, a);
      }
      g[4 * i + j] = a;
    }
#pragma unroll
  for (int i = 12; i < 16; ++i) g[i] = 0;
}
template <typename F> __device__ __forceinline__ void flip_sums(F (&g)[16], uint32_t p) {
#pragma unroll
  for (int e = 0; e < 12; ++e)
    if (odd_entry(e)) g[e] = flip_sign(g[e], p);
}
// A stage's matrices on its 16 values.
template <typename F>
__device__ __forceinline__ void stage_values(F (&v)[16], const PTab<F>& tb, uint32_t g0, const FrameStage& st) {
  F c[12];
  load12(tb.m[0], c);
  if (st.ng == 2) {
    const uint32_t p = y_parity(g0);
    flip_odd(c, p);
    apply_m<1, true>(v, c);
    load12(tb.m[1], c);
    flip_odd(c, p);
    apply_m<4, true>(v, c);
  } else {
    column_signs(v, g0, st);
    apply_m<1, false>(v, c);
    column_signs(v, g0, st);
  }
}

template <typename F, int LT>
__device__ __forceinline__ void pass_tables(const FrameStage* __restrict__ st, int nst, const F* __restrict__ bm, PTab<F>* tab) {
  for (int i = threadIdx.x; i < nst * 24; i += 1 << LT) {
    const FrameStage& s = st[i / 24];
    const int e = i % 24, w = e / 12, c = e - 12 * w, r = c / 4 + 1, k = c & 3;
    F v = r == k ? F(1) : F(0);
    if (w < s.ng) {
      const F* m = bm + 2 * s.off[2 * w];
      const int kind = s.diag >> (4 * w) & 3;
      if (kind == 0) v = m[c];
      else if (kind == 1 && (r & 1) && (k & 1)) v = m[(r & 2) + (k >> 1)];  // X, Y block
      else if (kind == 2 && r == k && r > 1) v = F(-1);
    }
    tab[i / 24].m[w][c] = v;
  }
}

// Tile-independent tables of a pass: thread bases, slot offsets (shared and
// global) and the threads' global parts.
template <int LT>
__device__ __forceinline__ void pauli_setup(const FrameStage* __restrict__ st, int nst, uint16_t* tbs, uint32_t* soff,
                                            uint32_t* gso, uint32_t* tg) {
  pass_setup<LT>(st, nst, tbs, soff);
  const uint32_t tid = threadIdx.x;
  for (int i = tid; i < nst * 16; i += 1 << LT) gso[i] = slot_xor(st[i >> 4].ge, i & 15);
  for (int k = 0; k < nst; ++k) {
    uint32_t b = 0;
#pragma unroll
    for (int i = 0; i < LT; ++i)
      if (tid >> i & 1u) b ^= st[k].gtv[i];
    tg[k * (1 << LT) + tid] = b;
  }
}
template <typename F> __host__ __device__ constexpr size_t pauli_tables(int nst, int threads) {
  return static_cast<size_t>(nst) * (sizeof(PTab<F>) + 32 * sizeof(uint32_t) + threads * sizeof(uint32_t)) + tb_bytes(nst, threads);
}

// One forward pass, `in` to `out` (the same buffer: in place).  Bound by
// instruction issue (51 to 65% of its slots; 18 instructions a value and stage, 6
// of them FMAs) and shared-memory wavefronts (18 stages of 107 conflict) with DRAM
// at 30 to 40%.  12 qubits, 8 layers, complex64, value and gradient: 19.3 -> 6.7 ms
// a call (32 passes of 47 to 56 us forward, twice, and of 105 us back, against 61
// of 110 us and reverse steps of 200 us on matrix entries); 7 qubits, 5 layers,
// complex128, 16 sets: 3.9 -> 0.45 ms.  Signs in the matrices instead of on the
// values and the first tables formed before the wait: 6.94 -> 6.72 ms.
template <typename F, int T, int MINB>
__global__ void __launch_bounds__(1 << (T - 4), MINB)
    k_pauli_fwd(const F* in, F* out, const PassArg P, const FrameStage* __restrict__ stages, const F* __restrict__ bmat,
                int64_t bstride, int batch, int rev, int first) {
  constexpr int LT = T - 4, NT = 1 << LT;
  constexpr uint32_t TB = sizeof(F) << T;
  const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  PTab<F>* tab = reinterpret_cast<PTab<F>*>(smem + 2 * TB);
  uint32_t* soff = reinterpret_cast<uint32_t*>(tab + P.nst);
  uint32_t* gso = soff + 16 * P.nst;
  uint32_t* tg = gso + 16 * P.nst;
  uint16_t* tbs = reinterpret_cast<uint16_t*>(tg + NT * P.nst);
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  if (!first) asm volatile("griddepcontrol.launch_dependents;");
  const FrameStage* st = stages + P.st0;
  const int nst = P.nst;
  pauli_setup<LT>(st, nst, tbs, soff, gso, tg);
  const uint32_t opos_lane = P.opos[lane];
  const bool on = (lane >> 2) < static_cast<uint32_t>(nst);
  const uint32_t r_lane = on ? st[lane >> 2].r[lane & 3] : 0u;
  const TileCopy<F, LT> copy(P);
  const uint64_t tiles_per = 1ULL << P.nouter;
  const int64_t ntiles = static_cast<int64_t>(tiles_per) * batch;
  const uint64_t rmask = rev ? tiles_per - 1 : 0;
  auto rep_of = [&](int64_t tl) {
    return tile_rep((static_cast<uint64_t>(tl) & (tiles_per - 1)) ^ rmask, opos_lane, P.nouter);
  };
  auto load = [&](uint32_t dst, int64_t tl) {
    const F* src = in + ((tl >> P.nouter) << P.nb);
    copy.each(P, rep_of(tl), dst, [&](uint32_t a, uint32_t b) { cp_async16(sbase + b, src + a); });
  };
  // The first pass of a call may start before prep has written the matrices: it waits,
  // and only then lets the second start.  From there on the matrices need no
  // wait, the states do.
  int64_t last = -1;
  if (first) asm volatile("griddepcontrol.wait;\n griddepcontrol.launch_dependents;" ::: "memory");
  if (blockIdx.x < ntiles) {
    last = static_cast<int64_t>(blockIdx.x) >> P.nouter;
    pass_tables<F, LT>(st, nst, bmat + last * bstride, tab);
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
    const uint32_t rep = rep_of(tile);
    const uint32_t flips = __ballot_sync(0xffffffffu, (__popc(rep & r_lane) & 1u) != 0u);
    if (inst != last) {
      pass_tables<F, LT>(st, nst, bmat + inst * bstride, tab);
      last = inst;
    }
    cp_wait<1>();
    __syncthreads();
    F* g = out + (inst << P.nb);
    for (int k = 0; k < nst; ++k) {
      const uint32_t nib = (flips >> (4 * k)) & 15u;
      const uint32_t* so = soff + 16 * k;
      const uint32_t e[4] = {so[1], so[2], so[4], so[8]};
      const uint32_t base = s ^ (static_cast<uint32_t>(tbs[k * NT + tid]) << 2) ^ so[nib];
      const uint32_t g0 = rep ^ tg[k * NT + tid] ^ gso[16 * k + nib];
      uint32_t a[16];
      F v[16];
      slot_offsets(e, base, a);
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = lds<F>(a[j]);
      stage_values(v, tab[k], g0, st[k]);
      if (P.direct && k + 1 == nst) {
        const uint32_t ge[4] = {gso[16 * k + 1], gso[16 * k + 2], gso[16 * k + 4], gso[16 * k + 8]};
        slot_offsets(ge, g0, a);
#pragma unroll
        for (int j = 0; j < 16; ++j) g[a[j]] = v[j];
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) sts(a[j], v[j]);
        __syncthreads();
      }
    }
    if (!P.direct)
      copy.each(P, rep, s, [&](uint32_t a, uint32_t b) { *reinterpret_cast<float4*>(g + a) = lds<float4>(b); });
    __syncthreads();
    s ^= TB;
  }
}

// One reverse pass: the input of every stage is kept in shared memory by a
// forward walk over the tile; backwards, each wire's cotangent (entries of lambda
// after its matrix times entries of the values before it, the other wire's matrix
// on one side) is summed, in type A in a thread and a warp, in float64 across warps
// and tiles, and lambda goes through the transposed matrices.
// Not launched ahead of the previous pass: two of these on an SM at once take each
// other's L2 (12 qubits 7.08 instead of 6.72 ms).
template <typename F, typename A, int T, int MINB>
__global__ void __launch_bounds__(1 << (T - 4), MINB)
    k_pauli_bwd(const F* __restrict__ xin, F* __restrict__ lam, const PassArg P, const FrameStage* __restrict__ stages,
                const F* __restrict__ bmat, int64_t bstride, double* __restrict__ gacc, int64_t gstride, int batch) {
  constexpr int LT = T - 4, NT = 1 << LT, NW = NT / 32;
  constexpr uint32_t TB = sizeof(F) << T;
  const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int nst = P.nst;
  const uint32_t lt = static_cast<uint32_t>(nst) * TB;  // lambda's tile, after the stage inputs
  PTab<F>* tab = reinterpret_cast<PTab<F>*>(smem + lt + TB);
  uint32_t* soff = reinterpret_cast<uint32_t*>(tab + nst);
  uint32_t* gso = soff + 16 * nst;
  uint32_t* tg = gso + 16 * nst;
  uint16_t* tbs = reinterpret_cast<uint16_t*>(tg + NT * nst);
  double* sacc = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(tbs) + tb_bytes(nst, NT));
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const FrameStage* st = stages + P.st0;
  pauli_setup<LT>(st, nst, tbs, soff, gso, tg);
  for (int i = tid; i < NW * nst * 32; i += NT) sacc[i] = 0.0;
  const uint32_t opos_lane = P.opos[lane];
  const bool on = (lane >> 2) < static_cast<uint32_t>(nst);
  const uint32_t r_lane = on ? st[lane >> 2].r[lane & 3] : 0u;
  const TileCopy<F, LT> copy(P);
  const uint64_t tiles_per = 1ULL << P.nouter;
  const int64_t ntiles = static_cast<int64_t>(tiles_per) * batch;
  int64_t last = -1;
  auto flush = [&](int64_t inst) {
    if (!gacc) return;
    for (int i = tid; i < nst * 24; i += NT) {
      const int k = i / 24, e = i - 24 * k, w = e / 12, c = e - 12 * w, gt = w < st[k].ng ? st[k].gate[2 * w] : -1;
      if (gt < 0) continue;
      double x = 0.0;
      for (int q = 0; q < NW; ++q) x += sacc[(q * nst + k) * 32 + 16 * w + c];
      atomicAdd(&gacc[inst * gstride + 12 * gt + c], x);
    }
  };
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t inst = tile >> P.nouter, ibase = inst << P.nb;
    const uint32_t rep = tile_rep(static_cast<uint64_t>(tile) & (tiles_per - 1), opos_lane, P.nouter);
    const uint32_t flips = __ballot_sync(0xffffffffu, (__popc(rep & r_lane) & 1u) != 0u);
    __syncthreads();
    copy.each(P, rep, 0, [&](uint32_t a, uint32_t b) {
      cp_async16(sbase + b, xin + ibase + a);
      cp_async16(sbase + lt + b, lam + ibase + a);
    });
    cp_commit();
    if (inst != last) {
      if (last >= 0) {
        flush(last);
        __syncthreads();
        for (int i = tid; i < NW * nst * 32; i += NT) sacc[i] = 0.0;
      }
      pass_tables<F, LT>(st, nst, bmat + inst * bstride, tab);
      last = inst;
    }
    cp_wait<0>();
    __syncthreads();
    auto slots = [&](int k, uint32_t (&a)[16]) {
      const uint32_t nib = (flips >> (4 * k)) & 15u;
      const uint32_t* so = soff + 16 * k;
      const uint32_t e[4] = {so[1], so[2], so[4], so[8]};
      slot_offsets(e, (static_cast<uint32_t>(tbs[k * NT + tid]) << 2) ^ so[nib], a);
      return rep ^ tg[k * NT + tid] ^ gso[16 * k + nib];
    };
    for (int k = 0; k + 1 < nst; ++k) {
      uint32_t a[16];
      const uint32_t g0 = slots(k, a);
      F v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = lds<F>(k * TB + a[j]);
      stage_values(v, tab[k], g0, st[k]);
#pragma unroll
      for (int j = 0; j < 16; ++j) sts(k * TB + TB + a[j], v[j]);
      __syncthreads();
    }
    for (int k = nst - 1; k >= 0; --k) {
      const PTab<F>& tb = tab[k];
      uint32_t a[16];
      const uint32_t g0 = slots(k, a);
      F l[16], c[12];
#pragma unroll
      for (int j = 0; j < 16; ++j) l[j] = lds<F>(lt + a[j]);
      double* acc = sacc + (warp * nst + k) * 32;
      const bool wa = gacc && st[k].gate[0] >= 0, wb = gacc && st[k].ng > 1 && st[k].gate[2] >= 0;
      auto add = [&](double* to, A (&g)[16]) {
        const A t = warp_rs16(g, lane);
        if (!(lane & 1u)) to[lane >> 1] += static_cast<double>(t);
      };
      F x[16];
      if (wa || wb) {
#pragma unroll
        for (int j = 0; j < 16; ++j) x[j] = lds<F>(k * TB + a[j]);
      }
      if (st[k].ng == 2) {
        const uint32_t p = y_parity(g0);
        A g[16];
        if (wb) {
          F y[16];
          load12(tb.m[0], c);
          flip_odd(c, p);
#pragma unroll
          for (int j = 0; j < 16; ++j) y[j] = x[j];
          apply_m<1, true>(y, c);
          outer_sum<4, true>(l, y, g);
          flip_sums(g, p);
          add(acc + 16, g);
        }
        load12(tb.m[1], c);
        flip_odd(c, p);
        apply_mt<4, true>(l, c);
        if (wa) {
          outer_sum<1, true>(l, x, g);
          flip_sums(g, p);
          add(acc, g);
        }
        load12(tb.m[0], c);
        flip_odd(c, p);
        apply_mt<1, true>(l, c);
      } else {
        column_signs(l, g0, st[k]);
        if (wa) {
          A g[16];
          column_signs(x, g0, st[k]);
          outer_sum<1, false>(l, x, g);
          add(acc, g);
        }
        load12(tb.m[0], c);
        apply_mt<1, false>(l, c);
        column_signs(l, g0, st[k]);
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) sts(lt + a[j], l[j]);
      __syncthreads();
    }
    copy.each(P, rep, 0, [&](uint32_t a, uint32_t b) {
      *reinterpret_cast<float4*>(lam + ibase + a) = lds<float4>(lt + b);
    });
  }
  __syncthreads();
  if (last >= 0) flush(last);
}

// ---- parameters and chain rule, float64 ------------------------------------
// Rows X, Z, Y of transfer matrices (row I is (1, 0, 0, 0)).
__device__ void pauli2(int k, double2* p) {  // I, X, Z, Y
  m_zero(p, 2);
  if (k == 0) { p[0].x = 1; p[3].x = 1; }
  else if (k == 1) { p[1].x = 1; p[2].x = 1; }
  else if (k == 2) { p[0].x = 1; p[3].x = -1; }
  else { p[1].y = -1; p[2].y = 1; }
}
// m[r][c] = Re tr(P_r A P_c B^dagger) * f
__device__ void transfer_of(const double2* A, const double2* B, double f, double* m) {
  for (int c = 0; c < 4; ++c) {
    double2 p[4], t[4], x[4];
    pauli2(c, p);
    m_mul(A, p, t, 2);
    m_mul_bh(t, B, x, 2);
    m[c] = f * (x[1].x + x[2].x);
    m[4 + c] = f * (x[0].x - x[3].x);
    m[8 + c] = f * (x[2].y - x[1].y);
  }
}
__device__ void prim_transfer(const DevPrim& p, const DevOp* ops, const double* ang, const double2* cpool, double* m) {
  if (p.form != PF_CONST) {
    double2 u[4], tmp[4];
    op_matrix(ops[p.op], ang, nullptr, u, -1, tmp);
    transfer_of(u, u, 0.5, m);
    return;
  }
  // constant superoperator on (ket, bra): the image of P_c, traced with P_r
  const double2* S = cpool + p.const_off;
  for (int c = 0; c < 4; ++c) {
    double2 q[4], x[4];
    pauli2(c, q);
    for (int s = 0; s < 4; ++s) {
      x[s] = make_double2(0, 0);
      for (int t = 0; t < 4; ++t) x[s] = cfma(S[4 * s + t], q[t], x[s]);
    }
    m[c] = 0.5 * (x[1].x + x[2].x);
    m[4 + c] = 0.5 * (x[0].x - x[3].x);
    m[8 + c] = 0.5 * (x[2].y - x[1].y);
  }
}
// o = a b
__device__ void transfer_mul(const double* a, const double* b, double* o) {
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 4; ++c) {
      double v = c == 0 ? a[4 * r] : 0.0;
      for (int k = 0; k < 3; ++k) v = fma(a[4 * r + k + 1], b[4 * k + c], v);
      o[4 * r + c] = v;
    }
}

template <typename F>
__global__ void k_pauli_prep(const FrameGate* __restrict__ gates, int ngates, const DevBlock* __restrict__ blocks,
                             const DevPrim* __restrict__ prims, const DevOp* __restrict__ ops,
                             const double* __restrict__ angles, int n_angles, const double2* __restrict__ cpool,
                             F* __restrict__ bmat, int64_t bstride, int batch, F* __restrict__ state, int nb) {
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<int64_t>(batch) * ngates) return;
  const int64_t inst = idx / ngates;
  const FrameGate fg = gates[idx - inst * ngates];
  if (fg.diag == 2) return;
  const DevBlock blk = blocks[fg.block];
  const double* ang = angles ? angles + inst * n_angles : nullptr;
  double acc[12], pm[12], tmp[12];
  prim_transfer(prims[blk.prim_begin], ops, ang, cpool, acc);
  for (int p = blk.prim_begin + 1; p < blk.prim_end; ++p) {
    prim_transfer(prims[p], ops, ang, cpool, pm);
    transfer_mul(pm, acc, tmp);
    for (int i = 0; i < 12; ++i) acc[i] = tmp[i];
  }
  // A NaN or infinite angle: not every word's value depends on this gate, but the
  // density matrix has no finite entry left.  The coefficient of the identity, that
  // no pass writes, tells k_pauli_expval; through the first columns of the
  // matrices' cotangents it reaches every gradient.
  double all = 0.0;
  for (int i = 0; i < 12; ++i) all += acc[i];
  if (!isfinite(all)) state[inst << nb] = static_cast<F>(all - all);
  F* o = bmat + inst * bstride + 2 * fg.mat_off;
  if (fg.diag == 1) {
    o[0] = static_cast<F>(acc[1]);
    o[1] = static_cast<F>(acc[3]);
    o[2] = static_cast<F>(acc[9]);
    o[3] = static_cast<F>(acc[11]);
    return;
  }
  for (int i = 0; i < 12; ++i) o[i] = static_cast<F>(acc[i]);
}

// Block cotangent -> angles: prefix products forwards, the cotangent through the
// transposed prims backwards.
__global__ void k_pauli_chain(const FrameGate* __restrict__ gates, int ngates, const DevBlock* __restrict__ blocks,
                              const DevPrim* __restrict__ prims, const DevOp* __restrict__ ops,
                              const double* __restrict__ angles, int n_angles, const double2* __restrict__ cpool,
                              const double* __restrict__ gacc, int64_t gstride, int batch, double* __restrict__ grad) {
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<int64_t>(batch) * ngates) return;
  const int64_t inst = idx / ngates;
  const FrameGate fg = gates[idx - inst * ngates];
  if (fg.grad < 0) return;
  const DevBlock blk = blocks[fg.block];
  const double* ang = angles + inst * n_angles;
  double* out = grad + inst * n_angles;
  const int m = blk.prim_end - blk.prim_begin;
  double pre[kMaxFusePrims][12], P[12], X[12], t[12];
  // pre[i]: product of the prims before i (i >= 1)
  for (int i = 0; i + 1 < m; ++i) {
    prim_transfer(prims[blk.prim_begin + i], ops, ang, cpool, P);
    if (i == 0)
      for (int e = 0; e < 12; ++e) pre[1][e] = P[e];
    else
      transfer_mul(P, pre[i], pre[i + 1]);
  }
  const double* g = gacc + inst * gstride + 12 * fg.grad;
  for (int e = 0; e < 12; ++e) X[e] = g[e];
  for (int i = m - 1; i >= 0; --i) {
    const DevPrim pr = prims[blk.prim_begin + i];
    if (pr.form != PF_CONST && ops[pr.op].grad && ops[pr.op].n_angles > 0) {
      const DevOp op = ops[pr.op];
      double2 u[4], du[4], tmp[4];
      op_matrix(op, ang, nullptr, u, -1, tmp);
      for (int j = 0; j < op.n_angles; ++j) {
        op_matrix(op, ang, nullptr, du, j, tmp);
        transfer_of(du, u, 1.0, P);  // Re tr(P_r dU P_c U^dagger): both sides' halves
        double v = 0.0;
        if (i == 0) {
          for (int e = 0; e < 12; ++e) v = fma(X[e], P[e], v);
        } else {
          transfer_mul(P, pre[i], t);
          for (int e = 0; e < 12; ++e) v = fma(X[e], t[e], v);
        }
        atomicAdd(&out[op.angle_slot + j], v);
      }
    }
    if (i == 0) break;
    prim_transfer(pr, ops, ang, cpool, P);
    for (int k = 0; k < 3; ++k)
      for (int c = 0; c < 4; ++c) {
        double v = 0.0;
        for (int r = 0; r < 3; ++r) v = fma(P[4 * r + k + 1], X[4 * r + c], v);
        t[4 * k + c] = v;
      }
    for (int e = 0; e < 12; ++e) X[e] = t[e];
  }
}

// |0..0><0..0|: coefficient 1 on every word without X or Y
template <typename F> __global__ void k_pauli_init(F* __restrict__ s, int64_t total, uint32_t xmask) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    s[i] = (static_cast<uint32_t>(i) & xmask) == 0 ? F(1) : F(0);
}
template <typename F>
__global__ void k_pauli_expval(const F* __restrict__ s, int nb, const PauliObs* __restrict__ obs, int n_obs, int batch,
                               double* __restrict__ out) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<int64_t>(n_obs) * batch) return;
  const int64_t inst = i / n_obs;
  const PauliObs o = obs[i - inst * n_obs];
  const F one = s[inst << nb];  // NaN: see k_pauli_prep
  out[i] = one != one ? static_cast<double>(one) : o.coeff * static_cast<double>(s[(inst << nb) + o.index]);
}
template <typename F>
__global__ void k_pauli_seed(F* __restrict__ lam, int nb, const PauliObs* __restrict__ obs, int n_obs, int batch,
                             const double* __restrict__ ct, double* __restrict__ gacc, int64_t gstride) {
  const int64_t inst = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (inst >= batch) return;
  // one thread an instance: words may coincide
  bool finite = true;
  for (int o = 0; o < n_obs; ++o) {
    F* p = lam + (inst << nb) + obs[o].index;
    const double w = obs[o].coeff * ct[inst * n_obs + o];
    finite = finite && isfinite(w);
    *p = static_cast<F>(static_cast<double>(*p) + w);
  }
  // a cotangent that is not finite leaves no entry of lambda's matrix finite, and
  // so no gradient of the instance, also where its word does not reach a gate
  if (!finite && gacc)
    for (int64_t i = 0; i < gstride; ++i) gacc[inst * gstride + i] = __longlong_as_double(0x7ff8000000000000LL);
}

template <typename F, int T> constexpr int fwd_ctas() { return sizeof(F) == 4 ? (T == 11 ? 8 : 16) : (T == 11 ? 5 : 10); }
template <typename F, typename A, int T> constexpr int bwd_ctas() {
  return sizeof(A) == 4 ? 4 : sizeof(F) == 4 ? (T == 11 ? 3 : 6) : (T == 11 ? 2 : 4);
}

template <typename F> size_t fwd_smem(const FramePass& p) {
  return (static_cast<size_t>(2) << p.t) * sizeof(F) + pauli_tables<F>(p.nst, 1 << (p.t - 4));
}
template <typename F> size_t bwd_smem(const FramePass& p) {
  const int nt = 1 << (p.t - 4);
  return (static_cast<size_t>(p.nst + 1) << p.t) * sizeof(F) + pauli_tables<F>(p.nst, nt) +
         static_cast<size_t>(nt / 32) * p.nst * 32 * sizeof(double);
}
template <typename F> const void* fwd_kernel(const FramePass& p) {
  return p.t == 10 ? reinterpret_cast<const void*>(&k_pauli_fwd<F, 10, fwd_ctas<F, 10>()>)
                   : reinterpret_cast<const void*>(&k_pauli_fwd<F, 11, fwd_ctas<F, 11>()>);
}
// Cotangent sums below 2^16 coefficients (seven qubits) are float64 from the product
// on, as in the general reverse pass of that size; larger ones are summed in the
// run precision, as in the specialised reverse steps.
template <typename F, typename A, int T> const void* bwd_of() {
  return reinterpret_cast<const void*>(&k_pauli_bwd<F, A, T, bwd_ctas<F, A, T>()>);
}
template <typename F> const void* bwd_kernel(const FramePass& p, int nb) {
  if (p.t == 10) return bwd_of<F, double, 10>();  // five qubits
  return nb < 16 ? bwd_of<F, double, 11>() : bwd_of<F, F, 11>();
}

template <typename F> int upload_shapes(const FramePlan& fp, int nb, FrameDev* d) {
  for (const FramePass& p : fp.passes)
    for (int rev = 0; rev < 2; ++rev) {
      const void* k = rev ? bwd_kernel<F>(p, nb) : fwd_kernel<F>(p);
      JQ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
      int n = 0;
      JQ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, 1 << (p.t - 4), rev ? bwd_smem<F>(p) : fwd_smem<F>(p)));
      (rev ? d->adj_ctas : d->fwd_ctas).push_back(std::max(1, n));
    }
  return JQ_OK;
}

template <typename F>
int pass_fwd(const jq_plan* plan, const FrameDev& d, size_t i, const F* in, F* out, int batch, const F* bmat, int sms,
             cudaStream_t st, bool pdl) {
  const FramePass& p = plan->pauli.passes[i];
  PassArg a = pass_arg(p, plan->n_bits, false);
  const int64_t ntiles = (1LL << p.nouter) * batch;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(std::min<int64_t>(ntiles, static_cast<int64_t>(sms) * d.fwd_ctas[i])));
  cfg.blockDim = dim3(1u << (p.t - 4));
  cfg.dynamicSmemBytes = fwd_smem<F>(p);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  const FrameStage* sp = d.stages;
  int64_t bs = 2 * plan->bmat_stride;
  int rev = static_cast<int>(i & 1), first = i == 0;
  void* args[] = {&in, &out, &a, &sp, &bmat, &bs, &batch, &rev, &first};
  JQ_CUDA(cudaLaunchKernelExC(&cfg, fwd_kernel<F>(p), args));
  return JQ_OK;
}

unsigned blocks_for(int64_t work, int threads) { return static_cast<unsigned>((work + threads - 1) / threads); }

template <typename F>
int start(const jq_plan* plan, const FrameDev& d, const DeviceTables& T, int batch, const double* angles, F* bmat, F* s,
          int sms, cudaStream_t st) {
  const int64_t total = static_cast<int64_t>(batch) << plan->n_bits;
  k_pauli_init<F><<<std::min<unsigned>(blocks_for(total, 256), static_cast<unsigned>(sms) * 16), 256, 0, st>>>(
      s, total, 0x55555555u & ((1u << plan->n_bits) - 1u));
  const int ng = static_cast<int>(plan->pauli.gates.size());
  if (ng > 0)
    k_pauli_prep<F><<<blocks_for(static_cast<int64_t>(ng) * batch, 64), 64, 0, st>>>(
        d.gates, ng, T.blocks, T.prims, T.ops, angles, plan->n_angles, reinterpret_cast<const double2*>(T.const_pool),
        bmat, 2 * plan->bmat_stride, batch, s, plan->n_bits);
  JQ_CUDA(cudaGetLastError());
  return JQ_OK;
}

template <typename F>
int forward_t(const jq_plan* plan, const FrameDev& d, const DeviceTables& T, int batch, const double* angles, F* s, F* bmat,
              double* out, int sms, cudaStream_t st) {
  int rc = start(plan, d, T, batch, angles, bmat, s, sms, st);
  if (rc) return rc;
  const bool pdl = pdl_on(st);
  for (size_t i = 0; i < plan->pauli.passes.size(); ++i)
    if ((rc = pass_fwd<F>(plan, d, i, s, s, batch, bmat, sms, st, pdl))) return rc;
  const int no = static_cast<int>(plan->pauli_obs.size());
  k_pauli_expval<F><<<blocks_for(static_cast<int64_t>(no) * batch, 128), 128, 0, st>>>(
      s, plan->n_bits, static_cast<const PauliObs*>(T.pauli_obs), no, batch, out);
  JQ_CUDA(cudaGetLastError());
  return JQ_OK;
}

template <typename F>
int backward_t(const jq_plan* plan, const FrameDev& d, const DeviceTables& T, int batch, const double* angles, F* bmat,
               double* gacc, F* lam, F* slots, int64_t n_slots, const double* ct, double* grad, int sms, cudaStream_t st) {
  const FramePlan& fp = plan->pauli;
  const int64_t P = static_cast<int64_t>(fp.passes.size());
  const size_t bytes = (sizeof(F) << plan->n_bits) * static_cast<size_t>(batch);
  const size_t step = ((bytes + 255) & ~static_cast<size_t>(255)) / sizeof(F);
  auto slot = [&](int64_t i) { return slots + step * static_cast<size_t>(i); };
  int rc = start(plan, d, T, batch, angles, bmat, slot(0), sms, st);
  if (rc) return rc;
  const bool pdl = pdl_on(st);
  // every pass input is kept where the slots allow it; otherwise the inputs of
  // each segment of S passes are recomputed from its checkpoint
  int64_t S = P;
  if (P > n_slots) {
    for (S = 1; S < P && (P + S - 1) / S + S > n_slots; ++S) {}
  }
  const int64_t nck = P > n_slots ? (P + S - 1) / S : 0;
  F* const seg0 = slot(nck);
  auto seg = [&](int64_t i) { return seg0 + step * static_cast<size_t>(i); };
  if (nck > 0)
    for (int64_t c = 0; c + 1 < nck; ++c)  // checkpoint c + 1 from c, through the segment's buffer
      for (int64_t p = c * S; p < (c + 1) * S; ++p)
        if ((rc = pass_fwd<F>(plan, d, static_cast<size_t>(p), p == c * S ? slot(c) : seg(0),
                              p + 1 == (c + 1) * S ? slot(c + 1) : seg(0), batch, bmat, sms, st, pdl)))
          return rc;
  JQ_CUDA(cudaMemsetAsync(lam, 0, bytes, st));
  const int no = static_cast<int>(plan->pauli_obs.size());
  const int64_t gstride = 12 * static_cast<int64_t>(fp.n_grad);
  const bool want = grad && fp.n_grad > 0;
  if (want) JQ_CUDA(cudaMemsetAsync(gacc, 0, sizeof(double) * gstride * batch, st));
  k_pauli_seed<F><<<blocks_for(batch, 64), 64, 0, st>>>(lam, plan->n_bits, static_cast<const PauliObs*>(T.pauli_obs), no,
                                                        batch, ct, want ? gacc : nullptr, gstride);
  JQ_CUDA(cudaGetLastError());
  for (int64_t c = std::max<int64_t>(nck, 1) - 1; c >= 0; --c) {
    const int64_t p0 = c * S, p1 = std::min(P, p0 + S);
    auto input = [&](int64_t p) { return nck > 0 ? (p == p0 ? slot(c) : seg(p - p0 - 1)) : slot(p); };
    for (int64_t p = p0; p + 1 < p1; ++p)
      if ((rc = pass_fwd<F>(plan, d, static_cast<size_t>(p), input(p), input(p + 1), batch, bmat, sms, st, pdl))) return rc;
    for (int64_t p = p1 - 1; p >= p0 && want; --p) {
      const FramePass& fpz = fp.passes[static_cast<size_t>(p)];
      PassArg a = pass_arg(fpz, plan->n_bits, true);
      const int64_t ntiles = (1LL << fpz.nouter) * batch;
      const FrameStage* sp = d.stages;
      int64_t bs = 2 * plan->bmat_stride;
      const F* xin = input(p);
      int64_t gs = gstride;
      void* args[] = {&xin, &lam, &a, &sp, &bmat, &bs, &gacc, &gs, &batch};
      JQ_CUDA(cudaLaunchKernel(
          bwd_kernel<F>(fpz, plan->n_bits),
          dim3(static_cast<unsigned>(std::min<int64_t>(ntiles, static_cast<int64_t>(sms) * d.adj_ctas[static_cast<size_t>(p)]))),
          dim3(1u << (fpz.t - 4)), args, bwd_smem<F>(fpz), st));
    }
  }
  if (grad && plan->n_angles > 0) JQ_CUDA(cudaMemsetAsync(grad, 0, sizeof(double) * plan->n_angles * batch, st));
  if (want) {
    const int ng = static_cast<int>(fp.gates.size());
    k_pauli_chain<<<blocks_for(static_cast<int64_t>(ng) * batch, 32), 32, 0, st>>>(
        d.gates, ng, T.blocks, T.prims, T.ops, angles, plan->n_angles, reinterpret_cast<const double2*>(T.const_pool), gacc,
        gstride, batch, grad);
    JQ_CUDA(cudaGetLastError());
  }
  return JQ_OK;
}

}  // namespace

int pauli_upload(const jq_plan* plan, FrameDev* d) {
  const FramePlan& fp = plan->pauli;
  if (!fp.on) return JQ_OK;
  int rc = frame_tables(fp, d);
  if (rc) return rc;
  return plan->dtype == JQ_C64 ? upload_shapes<float>(fp, plan->n_bits, d) : upload_shapes<double>(fp, plan->n_bits, d);
}

int pauli_forward(const jq_plan* plan, const DeviceTables& T, int batch, const double* angles, void* state, void* bmat,
                  double* out, int sm_count, cudaStream_t st) {
  return plan->dtype == JQ_C64 ? forward_t<float>(plan, T.pauli, T, batch, angles, static_cast<float*>(state),
                                                  static_cast<float*>(bmat), out, sm_count, st)
                               : forward_t<double>(plan, T.pauli, T, batch, angles, static_cast<double*>(state),
                                                   static_cast<double*>(bmat), out, sm_count, st);
}

int pauli_backward(const jq_plan* plan, const DeviceTables& T, int batch, const double* angles, void* bmat, double* gacc,
                   void* lam, void* slots, int64_t n_slots, const double* ct, double* grad_angles, int sm_count,
                   cudaStream_t st) {
  return plan->dtype == JQ_C64
             ? backward_t<float>(plan, T.pauli, T, batch, angles, static_cast<float*>(bmat), gacc, static_cast<float*>(lam),
                                 static_cast<float*>(slots), n_slots, ct, grad_angles, sm_count, st)
             : backward_t<double>(plan, T.pauli, T, batch, angles, static_cast<double*>(bmat), gacc, static_cast<double*>(lam),
                                  static_cast<double*>(slots), n_slots, ct, grad_angles, sm_count, st);
}

}  // namespace jq
