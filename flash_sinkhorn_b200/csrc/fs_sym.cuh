// Symmetric (Jacobi) Sinkhorn steps that evaluate every score entry ONCE for both potentials (fs_sym.cu).
#pragma once
#include "fs_common.cuh"
#include "fs_tc.cuh"

#include <cuda.h>

namespace fs {
namespace sym {

constexpr int kMaxProblems = 24;  // problems that advance in one launch (kernel parameters stay under 32 KB)

// Range record of one problem, kept on the device (see "Which steps" in fs_sym.cu). Values are floats encoded so
// that unsigned order is float order; every entry is a running maximum.
struct State {
  unsigned slot[3][8];  // per step modulo 3: {max u, -min u, max dlt, -min dlt} of the rows, then of the columns
  unsigned cst[4];      // max(-log2 a), max(log2 a), max(-log2 b), max(log2 b)
  unsigned range[kRangeWords];  // of the coordinates (OperandScales)
};

// What every kernel of a step needs to know about a problem. Cloud 0 = x, cloud 1 = y.
struct Geo {
  int n[2], nrt[2], nct[2], pad[2];  // points, row tiles of bm, column tiles of bn, padded points
  int bm, bn;
  int self;                          // one cloud against itself: only the tiles on one side of the diagonal
  int early;                         // 1: leave everything alone once ctrl->converged is set
  int by_tile;                       // column partials are one per row tile (not one per CTA and column tile)
  float ratio;                       // eps of the previous step / eps of this step
  OperandScales scales;              // of the fp16 coordinates
  State* st;
  Ctrl* ctrl;
  float* rp_m[2];  // one-sided steps: [column tile][row] offsets (log2 units) of the row sums of side c
  float* rp_s[2];  // [column tile][row] row sums; two-sided steps use side 0 only
  float* cp;       // two-sided steps: [piece][column] column sums
};

// One problem of a lockstep solve: caller's arrays, schedule-independent constants and the staged operands.
struct Problem {
  const float* src[2] = {nullptr, nullptr};
  const float* logw[2] = {nullptr, nullptr};
  const float* init[2] = {nullptr, nullptr};
  int n[2] = {0, 0};
  int d = 0, prec = 0;
  bool self = false;
  float cs_dot = 1.f, cs_sq = 1.f;  // cost scale of the dot term and of the squared norms (label cost: differ)
  LabelCost lab;
  // filled by layout()
  int kc = 0, kp = 0, kind = 0;
  float* opA[2];
  float* opB[2];
  float* pot[2];  // shifted potentials, updated in place
  float* sq[2];   // cost scale * squared norms
  Ctrl* ctrl;
  Geo geo;
  CUtensorMap map[8];  // per side: A-role full / tail, B-role full / tail
};

// Parameters of one step of one problem.
struct Step {
  Problem* p;
  double eps, eps_prev, eps_next;  // eps_next: eps of the step after this one (staged into the biases)
  float w, damp[2];
  bool early;
};

bool supported(int n, int m, int d, int prec, int nlab);
size_t bytes(int n, int m, int d, int prec, int nlab, bool self);
// Lays the problem out inside buf (bytes() of it) and encodes its tensor maps.
cudaError_t layout(Problem& p, char* buf);
// Operands, squared norms, initial potentials and the biases of a first step at eps0[i].
cudaError_t stage(Problem* const* p, const double* eps0, int cnt, cudaStream_t st);
// One step of cnt <= kMaxProblems problems of one feature dimension; t counts the steps since stage().
cudaError_t step(const Step* s, int cnt, int t, cudaStream_t st);
// Stages the biases again for a step at eps: steps that an early stop skipped have left those of their own.
cudaError_t rebias(const Problem& p, double eps, cudaStream_t st);
// out[c] = potential + squared-norm shift for both clouds (null pointers are skipped).
cudaError_t emit(Problem* const* p, float* const (*out)[2], int cnt, cudaStream_t st);

// Kernel of these sizes: 1 operands resident, 2 streamed in K chunks, 3 / 4 the same by tiles of 256 x 256 / 128 x 128.
int kernel_of(int n, int m, int d, int prec, int nlab);
// Two-sided steps that problems have taken on the current device (-1: error).
long long two_sided_steps();

int read_error_flag();
int clear_error_flag();

}  // namespace sym
}  // namespace fs
