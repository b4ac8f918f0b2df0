// Runs schedules of csrc/frame.cpp on the CPU, thread by thread and slot by slot
// as the kernels address them, against the circuit applied gate by gate.
//   frame_schedule_check <bits a gate: 1 or 2> <index bits> <tile bits> <low bits>
//                        <element bytes> <circuit kind 0..2> <seed>
// Kinds: 0 a ring of CX, 1 CX at growing range, 2 random permutations and gaps.
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../jaqsi_b200/csrc/frame.h"

using cd = std::complex<double>;
using jq::FrameOp;

namespace {

std::mt19937 rng;
int ri(int a, int b) { return a + static_cast<int>(rng() % static_cast<unsigned>(b - a + 1)); }

[[noreturn]] void fail(const char* what) {
  std::printf("%s\n", what);
  std::exit(1);
}

struct Circuit {
  std::vector<FrameOp> ops;
  std::vector<std::vector<cd>> mats;  // unitary 2x2, or real 4x4 on a wire's two bits
};

void add_gate(Circuit* c, int k, int wire) {
  std::normal_distribution<double> nd;
  const int d = 1 << k;
  FrameOp f;
  f.block = static_cast<int>(c->mats.size());
  f.k = k;
  for (int i = 0; i < k; ++i) f.bit[i] = k * wire + i;
  f.gate = {f.block, f.block * d * d, 0, 0, 0, 0};
  std::vector<cd> m(static_cast<size_t>(d * d));
  if (k == 1) {
    const double a = nd(rng), b = nd(rng), g = nd(rng);
    m = {std::polar(std::cos(a), b), std::polar(std::sin(a), g), -std::polar(std::sin(a), -g), std::polar(std::cos(a), -b)};
  } else {
    for (cd& x : m) x = 0.5 * nd(rng);
  }
  c->mats.push_back(m);
  c->ops.push_back(f);
}

// CX (control v, target w), SWAP or X; with two bits a wire CX adds the x bits
// forward and the z bits back.
void add_perm(Circuit* c, int k, int v, int w, int type) {
  FrameOp f;
  if (type == 2 && k == 1) {
    f.k = 1;
    f.bit[0] = v;
    f.col[0] = 1;
    f.b = 1;
    c->ops.push_back(f);
    return;
  }
  f.k = 2 * k;
  for (int i = 0; i < k; ++i) {
    f.bit[2 * i] = k * v + i;
    f.bit[2 * i + 1] = k * w + i;
  }
  const bool swap = type == 1;
  f.col[0] = swap ? 2 : 3;
  f.col[1] = swap ? 1 : 2;
  if (k == 2) {
    f.col[2] = swap ? 8 : 4;
    f.col[3] = swap ? 4 : 12;
  }
  c->ops.push_back(f);
}

void run_circuit(const Circuit& c, std::vector<cd>* x) {
  const size_t n = x->size();
  for (const FrameOp& f : c.ops) {
    std::vector<cd> y(n);
    for (size_t i = 0; i < n; ++i) {
      size_t rest = i, l = 0, from = 0;
      for (int q = 0; q < f.k; ++q) {
        if (i >> f.bit[q] & 1) { l ^= f.col[q]; from |= size_t(1) << q; }
        rest &= ~(size_t(1) << f.bit[q]);
      }
      auto at = [&](size_t local) {
        size_t j = rest;
        for (int q = 0; q < f.k; ++q)
          if (local >> q & 1) j |= size_t(1) << f.bit[q];
        return j;
      };
      if (f.block < 0) {
        y[at(l ^ f.b)] = (*x)[i];
      } else {
        const size_t d = size_t(1) << f.k;
        for (size_t r = 0; r < d; ++r) y[at(r)] += c.mats[static_cast<size_t>(f.block)][r * d + from] * (*x)[i];
      }
    }
    x->swap(y);
  }
}

uint32_t comb(const uint32_t* v, unsigned n, int bits) {
  uint32_t r = 0;
  for (int i = 0; i < bits; ++i)
    if (n >> i & 1) r ^= v[i];
  return r;
}

// The passes as the kernels run them: every address is checked to be in its tile
// and used once, every global index to be the one its shared address holds.
void run_passes(const jq::FramePlan& fp, const Circuit& c, int k, int elem, int max_st, std::vector<cd>* s) {
  for (const jq::FramePass& P : fp.passes) {
    const uint32_t size = 1u << P.t;
    if (P.nst < 1 || P.nst > max_st) fail("number of stages");
    std::vector<char> seen(s->size(), 0);
    for (uint64_t ti = 0; ti < (1ull << P.nouter); ++ti) {
      uint32_t rep = 0;
      for (int i = 0; i < P.nouter; ++i)
        if (ti >> i & 1) rep |= P.opos[i];
      std::vector<cd> sm(size);
      std::vector<uint32_t> where(size, ~0u);
      for (uint32_t l = 0; l < size; ++l) {
        const uint32_t g = rep ^ comb(P.g, l, P.t), a = comb(P.cs, l, P.t);
        if (g >= s->size() || seen[g]) fail("tiles overlap");
        if (a % static_cast<uint32_t>(elem) || a / elem >= size || where[a / elem] != ~0u) fail("shared offset of the copy");
        if (l < (1u << P.c) && g != (rep ^ l)) fail("low index bits");
        if (l && l * static_cast<uint32_t>(elem) < 16 && a != l * elem) fail("16-byte chunk");
        seen[g] = 1;
        sm[a / elem] = (*s)[g];
        where[a / elem] = g;
      }
      for (int st = 0; st < P.nst; ++st) {
        const jq::FrameStage& S = fp.stages[static_cast<size_t>(P.st0 + st)];
        unsigned nib = 0;
        for (int q = 0; q < 4; ++q)
          nib |= ((static_cast<unsigned>(__builtin_popcount(rep & S.r[q])) & 1u) ^ (S.sbits >> q & 1u)) << q;
        std::vector<char> hit(size, 0);
        for (uint32_t tid = 0; tid < size >> 4; ++tid) {
          const uint32_t base = comb(S.tv, tid, P.t - 4) ^ comb(S.e, nib, 4);
          const uint32_t gbase = rep ^ comb(S.gtv, tid, P.t - 4) ^ comb(S.ge, nib, 4);
          cd v[16];
          uint32_t at[16];
          for (unsigned j = 0; j < 16; ++j) {
            const uint32_t a = base ^ comb(S.e, j, 4);
            if (a % static_cast<uint32_t>(elem) || a / elem >= size || hit[a / elem]) fail("shared offset of a stage");
            hit[a / elem] = 1;
            at[j] = a / elem;
            if (where[at[j]] != (gbase ^ comb(S.ge, j, 4))) fail("global index of a slot");
            v[j] = sm[at[j]];
          }
          const unsigned d = 1u << k;
          for (int g = 0; g < S.ng; ++g) {
            const std::vector<cd>& m = c.mats[static_cast<size_t>(S.off[k * g]) / (d * d)];
            for (unsigned j = 0; j < 16; ++j) {
              if (j >> (k * g) & (d - 1)) continue;
              cd o[4] = {};
              for (unsigned r = 0; r < d; ++r)
                for (unsigned q = 0; q < d; ++q) o[r] += m[r * d + q] * v[j | q << (k * g)];
              for (unsigned r = 0; r < d; ++r) v[j | r << (k * g)] = o[r];
            }
          }
          for (unsigned j = 0; j < 16; ++j) sm[at[j]] = v[j];
        }
      }
      for (uint32_t a = 0; a < size; ++a) (*s)[where[a]] = sm[a];
    }
  }
}

}  // namespace

int main(int argc, char** argv) {
  if (argc != 8) fail("arguments");
  const int k = std::atoi(argv[1]), nb = std::atoi(argv[2]), t = std::atoi(argv[3]), low = std::atoi(argv[4]);
  const int elem = std::atoi(argv[5]), kind = std::atoi(argv[6]), wires = nb / k;
  rng.seed(static_cast<unsigned>(std::atoi(argv[7])));
  Circuit c;
  for (int layer = 0; layer < 5; ++layer) {
    for (int w = 0; w < wires; ++w)
      if (kind != 2 || ri(0, 3)) add_gate(&c, k, wires - 1 - w);
    for (int w = 0; w < wires; ++w) {
      const int v = (w + (kind == 1 ? layer % (wires - 1) + 1 : 1)) % wires;
      add_perm(&c, k, w, v, kind == 2 ? ri(0, 2) : 0);
    }
  }
  const int max_st = k == 2 ? (elem == 4 ? 6 : 5) : t == nb ? jq::kFrameMaxStages : jq::kFrameBallot;
  std::vector<uint64_t> zt;
  std::vector<double> sign;
  if (k == 1)
    for (int w = 0; w < nb; ++w) {
      zt.push_back(1 + rng() % ((uint64_t(1) << nb) - 1));
      sign.push_back(1.0);
    }
  const std::vector<uint64_t> words = zt;
  jq::FramePlan fp;
  if (!jq::frame_schedule(c.ops, nb, t, low, elem, max_st, &zt, &sign, &fp)) fail("no schedule");
  if (fp.gates.size() != c.mats.size()) fail("gates lost");
  std::normal_distribution<double> nd;
  std::vector<cd> x(size_t(1) << nb);
  for (cd& a : x) a = {nd(rng), k == 1 ? nd(rng) : 0.0};
  std::vector<cd> s = x;
  run_circuit(c, &x);
  run_passes(fp, c, k, elem, max_st, &s);
  double err = 0, norm = 0;
  if (k == 2) {  // coefficient l lies at the XOR of its bits' masks
    for (size_t l = 0; l < x.size(); ++l) {
      uint32_t p = 0;
      for (int b = 0; b < nb; ++b)
        if (l >> b & 1) p ^= fp.mask[static_cast<size_t>(b)];
      err = std::max(err, std::abs(s[p] - x[l]));
      norm = std::max(norm, std::abs(x[l]));
    }
  } else {
    for (size_t z = 0; z < words.size(); ++z) {
      double a = 0, b = 0;
      for (size_t i = 0; i < x.size(); ++i) {
        a += __builtin_parityll(i & words[z]) ? -std::norm(x[i]) : std::norm(x[i]);
        b += __builtin_parityll(i & zt[z]) ? -std::norm(s[i]) : std::norm(s[i]);
      }
      err = std::max(err, std::abs(a - sign[z] * b));
    }
    for (const cd& a : x) norm += std::norm(a);
  }
  std::printf("passes %zu stages %zu error %.1e\n", fp.passes.size(), fp.stages.size(), err / norm);
  // double arithmetic over at most a few hundred gates
  return err <= 1e-11 * norm ? 0 : 1;
}
