// Frame plans: statevector circuits of one-wire unitary gates and affine
// permutations (X, CX, SWAP and their products) run without moving an
// amplitude for a permutation.
//
// The state stays at fixed physical addresses; what a permutation changes is
// the frame, the affine map from a physical index p to the logical index:
// logical wire w of amplitude p is parity(p & r_w) ^ s_w, and flipping wire w
// moves p by XOR with the mask m_w.  A one-wire gate then acts on the pairs
// (p, p ^ m_w), the role of each half given by the functional r_w.  Gates a
// and b commute when r_a . m_b = r_b . m_a = 0.
//
// A pass holds the cosets of a t-dimensional subspace V of the index space
// (tile = one coset; V contains the lowest c unit vectors, so global accesses
// stay contiguous in runs of 2^c) and runs every gate whose mask lies in V.  A
// stage is up to four gates with r_i . m_j = delta_ij: a tensor product on
// four virtual qubits.  Register slots are spanned by the masks; thread bits
// by vectors on which all four functionals vanish, so that slot bit i is the
// role of gate i up to a per-tile flip that moves the stage's base address.
// Every address is XOR-linear in (tile, thread, slot).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "../../include/jqsim.h"

struct jq_plan;

namespace jq {

struct DevBlock;
struct DevPrim;
struct DevOp;
struct DeviceTables;

constexpr int kFrameMaxT = 12;      // largest tile (2^12 amplitudes)
constexpr int kFrameRB = 4;         // gates of a stage, register slots 2^4
constexpr int kFrameBallot = 8;     // stages of a pass with tile flips (4 ballot bits each)
constexpr int kFrameMaxStages = 24; // stages of a pass that holds the whole state

struct FrameGate {
  int32_t block;     // fused block of the plan
  int32_t mat_off;   // its parameters in the block-matrix row (run-dtype complex elements)
  int32_t diag;      // 1: diagonal block (statevectors: two elements, else four)
  int32_t grad;      // index among the gates with cotangents, -1: none wanted
  uint32_t m, r;     // mask and role functional
};

// Device descriptor of a stage.  Shared offsets are in
// bytes, swizzled.
struct FrameStage {
  uint32_t e[kFrameRB];               // shared offset of register vector q
  uint32_t tv[kFrameMaxT - kFrameRB]; // shared offset of thread bit i
  uint32_t ge[kFrameRB];              // the same vectors in global index space
  uint32_t gtv[kFrameMaxT - kFrameRB];
  uint32_t r[kFrameRB];               // role functional of gate q (0: no gate)
  uint32_t sbits;                     // bit q: role q inverted
  int32_t ng;                         // gates
  int32_t gate[kFrameRB];             // cotangent index of the gates, -1 none
  int32_t off[kFrameRB];              // mat_off of the gates, -1 none
  int32_t diag;                       // bits 2 q: FrameGate::diag of register bit q
};

struct FramePass {
  int32_t t = 0, c = 0;
  uint32_t cs[kFrameMaxT] = {};       // shared byte offset of copy vector g[i]
  int32_t st0 = 0, nst = 0;
  int32_t direct = 0;                 // last stage stores straight to global memory (whole sectors)
  int32_t adirect = 0;                // first stage (the adjoint's last) does
  uint32_t g[kFrameMaxT] = {};        // copy vectors: a basis of V, the lowest c unit vectors first
  int32_t nouter = 0;
  uint32_t opos[32] = {};             // global unit vector of tile-index bit i
};

struct FramePlan {
  bool on = false;
  std::vector<FrameGate> gates;
  int n_grad = 0;  // gates with cotangents
  std::vector<FrameStage> stages;
  std::vector<FramePass> passes;
  std::vector<uint32_t> mask;  // final mask of every logical bit
};

// Uploaded tables and launch shapes of a frame plan on one device.
struct FrameDev {
  FrameStage* stages = nullptr;
  FrameGate* gates = nullptr;
  std::vector<int> fwd_ctas, adj_ctas;  // CTAs an SM per pass
};

// A gate or an affine permutation in program order, as the planner sees it.
struct FrameOp {
  int block = -1;                 // >= 0: a gate on k = 1 or 2 bits (the same k in one schedule)
  int k = 0;
  int bit[8] = {};                // flat bit of local bit i
  uint32_t col[8] = {};           // permutation: P(x) = xor of col[i] over set bits ^ b
  uint32_t b = 0;
  FrameGate gate{};
};

// Schedules ops on nb index bits into passes of at most t_max bits that hold the
// lowest c bits, and at most max_st stages, for values of `elem` bytes.  zt / zsign:
// Z words over logical flat bits, rewritten to words over physical bits.  False
// when a size is out of range.
bool frame_schedule(const std::vector<FrameOp>& ops, int nb, int t_max, int c, int elem, int max_st,
                    std::vector<uint64_t>* zt, std::vector<double>* zsign, FramePlan* out);

int frame_upload(const jq_plan* plan, FrameDev* d);
int frame_tables(const FramePlan& fp, FrameDev* d);  // the tables alone
void frame_free(FrameDev* d);
// Arrays the gate matrices' kernel sets to zero for the kernels after it.
struct ZeroFill {
  double* p[2] = {nullptr, nullptr};
  int64_t n[2] = {0, 0};
};
int frame_prep(const jq_plan* plan, const FrameDev& d, const DevBlock* blocks, const DevPrim* prims, const DevOp* ops,
               const double* cpool, int batch, const double* angles, void* bmat, const ZeroFill& z, cudaStream_t st);
// from_zero: the states start at |0..0> and hold nothing yet (a plan with passes)
int frame_forward(const jq_plan* plan, const FrameDev& d, void* state, int batch, const void* bmat, bool from_zero,
                  int sm_count, cudaStream_t st);
// psi_in: final state (read by the first launched pass only), psi: workspace
// for the rest; gacc: 3 doubles a gate with cotangents, instance stride gstride doubles.
int frame_adjoint(const jq_plan* plan, const FrameDev& d, const void* psi_in, void* psi, void* lam, int batch,
                  const void* bmat, double* gacc, int64_t gstride, int sm_count, cudaStream_t st);
int frame_chain(const jq_plan* plan, const FrameDev& d, const DevBlock* blocks, const DevPrim* prims, const DevOp* ops,
                const double* cpool, int batch, const double* angles, const void* bmat, const double* gacc,
                int64_t gstride, double* grad_angles, cudaStream_t st);

// ---- noisy circuits in the Pauli basis (pauli.cu) -----------------------------
// An observable: coefficient `index` (physical, sign included) times coeff.
struct PauliObs {
  uint32_t index;
  double coeff;
};

int pauli_upload(const jq_plan* plan, FrameDev* d);
// state: the coefficients, half a density matrix's bytes.
int pauli_forward(const jq_plan* plan, const DeviceTables& T, int batch, const double* angles, void* state, void* bmat,
                  double* out, int sm_count, cudaStream_t st);
// gacc: 12 doubles a gate with cotangents; slots: n_slots >= 3 states of 256-byte
// aligned coefficients for pass inputs and checkpoints.
int pauli_backward(const jq_plan* plan, const DeviceTables& T, int batch, const double* angles, void* bmat, double* gacc,
                   void* lam, void* slots, int64_t n_slots, const double* ct, double* grad_angles, int sm_count,
                   cudaStream_t st);

}  // namespace jq
