// Host scheduler of frame plans (see frame.h).
#include "frame.h"

#include <algorithm>
#include <cstring>

namespace jq {
namespace {

int par64(uint64_t v) { return __builtin_popcountll(v) & 1; }

// A gate on n index bits: their masks, functionals and inversions.
struct Gate {
  int n = 0;
  uint32_t m[2] = {}, r[2] = {};
  int s[2] = {};
  FrameGate fg{};
};

bool commute(const Gate& a, const Gate& b) {
  for (int i = 0; i < a.n; ++i)
    for (int j = 0; j < b.n; ++j)
      if (par64(a.r[i] & b.m[j]) || par64(b.r[j] & a.m[i])) return false;
  return true;
}

// Span of GF(2) vectors by highest set bit.
struct Span {
  uint32_t v[32] = {};
  int dim = 0;
  uint32_t reduce(uint32_t x) const {
    while (x) {
      const int h = 31 - __builtin_clz(x);
      if (!v[h]) return x;
      x ^= v[h];
    }
    return 0;
  }
  bool add(uint32_t x) {
    x = reduce(x);
    if (!x) return false;
    v[31 - __builtin_clz(x)] = x;
    ++dim;
    return true;
  }
};

// Shared position of tile index l: 16-byte chunks (2^cb values) keep their
// order inside, the higher bits fold onto the three bank bits of a chunk.
uint32_t swizzle(uint32_t l, int cb) {
  uint32_t r = l;
  for (int pos = cb + 3; pos < 16; ++pos)
    if (l >> pos & 1u) r ^= 1u << (cb + (pos - cb) % 3);
  return r;
}

}  // namespace

bool frame_schedule(const std::vector<FrameOp>& ops, int nb, int t_max, int c, int elem, int max_st,
                    std::vector<uint64_t>* zt, std::vector<double>* zsign, FramePlan* out) {
  if (nb < kFrameRB || nb > 31 || t_max < kFrameRB || t_max > kFrameMaxT) return false;
  t_max = std::min(t_max, nb);
  c = std::min(c, t_max);
  if (c < 2) return false;  // chunks of 16 bytes are contiguous
  // `nbank` lane bits fill a shared-memory wavefront of amplitudes
  const int esh = elem == 4 ? 2 : elem == 8 ? 3 : 4, nbank = 7 - esh, cb = 4 - esh;
  // ---- gates in the frame ----------------------------------------------------
  std::vector<uint32_t> m(nb), r(nb);
  std::vector<int> s(nb, 0);
  for (int i = 0; i < nb; ++i) m[i] = r[i] = 1u << i;
  std::vector<Gate> gates;
  for (const FrameOp& op : ops) {
    if (op.block >= 0) {
      Gate g;
      g.n = op.k;
      for (int i = 0; i < op.k; ++i) {
        g.m[i] = m[op.bit[i]];
        g.r[i] = r[op.bit[i]];
        g.s[i] = s[op.bit[i]];
      }
      g.fg = op.gate;
      gates.push_back(g);
      continue;
    }
    // inverse of the linear part, by elimination on [A | I] (rows = outputs)
    const int k = op.k;
    uint32_t row[8] = {}, inv[8] = {};
    for (int o = 0; o < k; ++o) {
      for (int i = 0; i < k; ++i) row[o] |= (op.col[i] >> o & 1u) << i;
      inv[o] = 1u << o;
    }
    uint32_t a[8];
    std::copy(row, row + k, a);
    for (int i = 0; i < k; ++i) {
      int p = i;
      while (p < k && !(a[p] >> i & 1u)) ++p;
      if (p == k) return false;
      std::swap(a[p], a[i]);
      std::swap(inv[p], inv[i]);
      for (int o = 0; o < k; ++o)
        if (o != i && (a[o] >> i & 1u)) { a[o] ^= a[i]; inv[o] ^= inv[i]; }
    }
    // inv[i]: row i of A^-1 (over the new local bits)
    uint32_t rn[8], mn[8];
    int sn[8];
    for (int o = 0; o < k; ++o) {
      rn[o] = 0;
      mn[o] = 0;
      sn[o] = op.b >> o & 1u;
      for (int i = 0; i < k; ++i) {
        if (row[o] >> i & 1u) { rn[o] ^= r[op.bit[i]]; sn[o] ^= s[op.bit[i]]; }
        if (inv[i] >> o & 1u) mn[o] ^= m[op.bit[i]];  // (A^-1)[i][o]
      }
    }
    for (int o = 0; o < k; ++o) { r[op.bit[o]] = rn[o]; m[op.bit[o]] = mn[o]; s[op.bit[o]] = sn[o]; }
  }
  out->mask = m;
  // Z words over the logical bits -> words over the physical bits
  for (size_t z = 0; z < zt->size(); ++z) {
    uint64_t w = 0;
    for (int i = 0; i < nb; ++i)
      if ((*zt)[z] >> i & 1ULL) {
        w ^= r[i];
        if (s[i]) (*zsign)[z] = -(*zsign)[z];
      }
    (*zt)[z] = w;
  }
  // ---- passes ------------------------------------------------------------------
  const int ngate = static_cast<int>(gates.size());
  out->gates.clear();
  out->n_grad = 0;
  out->stages.clear();
  out->passes.clear();
  std::vector<int> rem(ngate);
  for (int i = 0; i < ngate; ++i) rem[i] = i;
  size_t head = 0;  // rem[head..] are left
  const int cap = kFrameRB / (gates.empty() ? 1 : gates[0].n);  // gates of a stage
  const size_t window = static_cast<size_t>(4 * nb);
  while (head < rem.size()) {
    Span V;
    for (int i = 0; i < c; ++i) V.add(1u << i);
    std::vector<std::vector<int>> stg;      // gates of each stage
    std::vector<int> deferred, members;
    size_t pos = head;
    for (; pos < rem.size() && deferred.size() <= window; ++pos) {
      const int g = rem[pos];
      bool ok = true;
      for (int d : deferred)
        if (!commute(gates[g], gates[d])) { ok = false; break; }
      Span U = V;
      if (ok) {
        for (int i = 0; i < gates[g].n; ++i) U.add(gates[g].m[i]);
        ok = U.dim <= t_max;
      }
      if (ok) {
        // earliest stage after the last one that holds a gate g must follow
        size_t k = stg.size();
        while (k > 0) {
          bool dual = true;
          for (int o : stg[k - 1])
            if (!commute(gates[g], gates[o])) { dual = false; break; }
          if (!dual) break;
          --k;
        }
        while (k < stg.size() && static_cast<int>(stg[k].size()) >= cap) ++k;
        if (k == stg.size() && static_cast<int>(stg.size()) >= max_st) ok = false;
        if (ok) {
          if (k == stg.size()) stg.emplace_back();
          stg[k].push_back(g);
          V = U;
          members.push_back(g);
        }
      }
      if (!ok) deferred.push_back(g);
    }
    // the gates left: the deferred ones, then those not looked at
    std::vector<int> left(deferred);
    left.insert(left.end(), rem.begin() + static_cast<std::ptrdiff_t>(pos), rem.end());
    rem.swap(left);
    head = 0;
    for (int b = 0; b < nb && V.dim < t_max; ++b) V.add(1u << b);
    // reduced basis: the lowest c unit vectors, then one vector per further
    // pivot (its lowest set bit), zero at every other pivot
    FramePass pd;
    pd.t = V.dim;
    pd.c = c;
    const int t = pd.t;
    std::vector<uint32_t> basis;
    std::vector<int> pivot;
    for (int i = 0; i < c; ++i) { basis.push_back(1u << i); pivot.push_back(i); }
    {
      for (int h = 0; h < 32; ++h)
        if (V.v[h]) {
          uint32_t x = V.v[h] & ~((1u << c) - 1u);
          for (size_t q = static_cast<size_t>(c); q < basis.size(); ++q)
            if (x >> pivot[q] & 1u) x ^= basis[q];
          if (!x) continue;
          const int p = __builtin_ctz(x);
          for (size_t q = static_cast<size_t>(c); q < basis.size(); ++q)
            if (basis[q] >> p & 1u) basis[q] ^= x;
          basis.push_back(x);
          pivot.push_back(p);
        }
    }
    if (static_cast<int>(basis.size()) != t) return false;
    uint32_t pmask = 0;
    for (int i = 0; i < t; ++i) pmask |= 1u << pivot[i];
    for (int b = 0; b < nb; ++b)
      if (!(pmask >> b & 1u)) pd.opos[pd.nouter++] = 1u << b;
    auto local = [&](uint32_t x) {
      uint32_t l = 0;
      for (int i = 0; i < t; ++i) l |= (x >> pivot[i] & 1u) << i;
      return l;
    };
    auto global = [&](uint32_t l) {
      uint32_t x = 0;
      for (int i = 0; i < t; ++i)
        if (l >> i & 1u) x ^= basis[i];
      return x;
    };
    auto bytes = [&](uint32_t l) { return swizzle(l, cb) << esh; };
    // copy vectors: the low unit vectors, then those whose shared offsets add
    // bank bits to the 8 lanes of a wavefront of 16-byte chunks
    {
      std::vector<uint32_t> left(basis.begin() + c, basis.end()), order(basis.begin(), basis.begin() + c);
      Span B;
      const uint32_t wm = 112u;
      for (uint32_t x : order) B.add(bytes(local(x)) & wm);
      while (!left.empty()) {
        size_t k = 0;
        for (size_t q = 0; q < left.size(); ++q)
          if (B.reduce(bytes(local(left[q])) & wm)) { k = q; break; }
        B.add(bytes(local(left[k])) & wm);
        order.push_back(left[k]);
        left.erase(left.begin() + static_cast<std::ptrdiff_t>(k));
      }
      for (int i = 0; i < t; ++i) { pd.g[i] = order[i]; pd.cs[i] = bytes(local(order[i])); }
    }
    // a stage whose functionals vanish on the lowest index bits can keep them as
    // lane bits: a warp's store then fills whole sectors.  Prefer such a stage
    // last (and, for the adjoint, first) where it commutes past the others.
    const int ns = 5 - esh;  // index bits of a 32-byte sector
    const uint32_t lowm = (1u << ns) - 1u;
    auto sector = [&](const std::vector<int>& st) {
      for (int g : st)
        for (int i = 0; i < gates[g].n; ++i)
          if (gates[g].r[i] & lowm) return false;
      return true;
    };
    auto passes_by = [&](size_t a, size_t b) {
      for (int x : stg[a])
        for (int y : stg[b])
          if (!commute(gates[x], gates[y])) return false;
      return true;
    };
    for (size_t k = stg.size(); k-- > 0;) {
      if (!sector(stg[k])) continue;
      bool ok = true;
      for (size_t q = k + 1; q < stg.size() && ok; ++q) ok = passes_by(k, q);
      if (!ok) continue;
      std::rotate(stg.begin() + static_cast<std::ptrdiff_t>(k), stg.begin() + static_cast<std::ptrdiff_t>(k) + 1, stg.end());
      break;
    }
    for (size_t k = 0; k + 1 < stg.size(); ++k) {
      if (!sector(stg[k])) continue;
      bool ok = true;
      for (size_t q = 0; q < k && ok; ++q) ok = passes_by(k, q);
      if (!ok) continue;
      std::rotate(stg.begin(), stg.begin() + static_cast<std::ptrdiff_t>(k), stg.begin() + static_cast<std::ptrdiff_t>(k) + 1);
      break;
    }
    pd.st0 = static_cast<int32_t>(out->stages.size());
    pd.nst = static_cast<int32_t>(stg.size());
    for (size_t k = 0; k < stg.size(); ++k) {
      FrameStage fs;
      std::memset(&fs, 0, sizeof(fs));
      fs.ng = static_cast<int32_t>(stg[k].size());
      uint32_t rho[kFrameRB] = {}, mu[kFrameRB] = {};
      for (int q = 0; q < kFrameRB; ++q) fs.gate[q] = fs.off[q] = -1;
      int ng = 0;  // register bits with a role
      for (int gi : stg[k]) {
        const Gate& g = gates[gi];
        FrameGate fg = g.fg;
        fg.m = g.m[0];
        fg.r = g.r[0];
        if (fg.grad >= 0) fg.grad = out->n_grad++;
        for (int i = 0; i < g.n; ++i, ++ng) {
          mu[ng] = local(g.m[i]);
          if (global(mu[ng]) != g.m[i]) return false;
          for (int q = 0; q < t; ++q) rho[ng] |= static_cast<uint32_t>(par64(g.r[i] & basis[q])) << q;
          fs.r[ng] = g.r[i];
          if (g.s[i]) fs.sbits |= 1u << ng;
          fs.gate[ng] = fg.grad;
          fs.off[ng] = fg.mat_off;
          fs.diag |= fg.diag << (2 * ng);
        }
        out->gates.push_back(fg);
      }
      // kernel of the functionals: projections of the unit vectors
      std::vector<uint32_t> kb;
      {
        Span S;
        for (int i = 0; i < t && static_cast<int>(kb.size()) < t - ng; ++i) {
          const uint32_t x = 1u << i;
          uint32_t y = x;
          for (int q = 0; q < ng; ++q)
            if (par64(rho[q] & x)) y ^= mu[q];
          if (y && S.add(y)) kb.push_back(y);
        }
        if (static_cast<int>(kb.size()) != t - ng) return false;
      }
      // lane bits first: vectors whose shared offsets differ on the bank bits
      const uint32_t bm = (1u << nbank) - 1u;
      std::vector<uint32_t> lanes, rest;
      {
        uint32_t ev[8] = {}, el[8] = {};  // echelon of bank parts and the vectors behind them
        int ne = 0;
        for (uint32_t x : kb) {
          uint32_t bx = swizzle(x, cb) & bm, y = x;
          for (int q = 0; q < ne; ++q)
            if (bx & (ev[q] & (~ev[q] + 1u))) { bx ^= ev[q]; y ^= el[q]; }
          if (bx && ne < nbank) {
            ev[ne] = bx;
            el[ne] = y;
            // keep the echelon reduced at the new pivot
            const uint32_t pv = bx & (~bx + 1u);
            for (int q = 0; q < ne; ++q)
              if (ev[q] & pv) { ev[q] ^= bx; el[q] ^= y; }
            ++ne;
            lanes.push_back(x);
          } else {
            rest.push_back(y);
          }
        }
      }
      std::vector<uint32_t> reg(mu, mu + ng);
      // register fillers: from the vectors that are not lanes, highest first
      for (int q = ng; q < kFrameRB; ++q) {
        if (!rest.empty()) { reg.push_back(rest.back()); rest.pop_back(); }
        else if (!lanes.empty()) { reg.push_back(lanes.back()); lanes.pop_back(); }
        else return false;
      }
      lanes.insert(lanes.end(), rest.begin(), rest.end());
      if (static_cast<int>(lanes.size()) != t - kFrameRB) return false;
      for (int q = 0; q < kFrameRB; ++q) { fs.e[q] = bytes(reg[q]); fs.ge[q] = global(reg[q]); }
      for (int i = 0; i < t - kFrameRB; ++i) { fs.tv[i] = bytes(lanes[i]); fs.gtv[i] = global(lanes[i]); }
      bool dir = t - kFrameRB >= ns;
      for (int i = 0; i < ns && dir; ++i) dir = fs.gtv[i] == 1u << i;
      if (k + 1 == stg.size()) pd.direct = dir;
      if (k == 0) pd.adirect = dir;
      out->stages.push_back(fs);
    }
    out->passes.push_back(pd);
  }
  out->on = true;
  return true;
}

}  // namespace jq
