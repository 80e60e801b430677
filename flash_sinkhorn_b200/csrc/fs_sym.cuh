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
  unsigned delta[2];    // early stop: largest move of a potential since the last check, checks taken in turn
  unsigned bar_count, bar_leave;  // grid barrier of the launches that this problem is the first of
};

// One step of one problem, in the problem's table on the device.
struct alignas(16) StepRec {
  float eps, eps_next, ratio, scale2;  // eps_next: of the step after this one (staged into the biases); ratio: eps of the
                                       // previous step / eps; scale2 = 2 cs log2e / eps
  float w, damp[2];
  unsigned todo;                       // kEmitPre | kEmitOut | kCheck | ordinal of the check << 8
};
constexpr unsigned kEmitPre = 1, kEmitOut = 2, kCheck = 4;  // write the potentials after this step to pre / out; early-stop test
// Records that a problem's table holds: 8 KB of its scratch, more steps than solves usually take. A longer solve goes on with a
// second launch behind an upload of the next 256.
constexpr int kTableSteps = 256;

// What every kernel of a step needs to know about a problem. Cloud 0 = x, cloud 1 = y.
struct Geo {
  int n[2], nrt[2], nct[2], pad[2];  // points, row tiles of bm, column tiles of bn, padded points
  int bm, bn;
  int self;                          // one cloud against itself: only the tiles on one side of the diagonal
  int by_tile;                       // column partials are one per row tile (not one per CTA and column tile)
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
  float* out[2] = {nullptr, nullptr};   // results of the steps that ask for them (null: not wanted)
  float* pre[2] = {nullptr, nullptr};
  float* snap[2] = {nullptr, nullptr};  // early stop: potentials at the last check
  Ctrl* ctrl;
  StepRec* table;        // of its own
  const StepRec* sched;  // table in use: its own, or that of a problem with the same steps
  Geo geo;
  CUtensorMap map[8];  // per side: A-role full / tail, B-role full / tail
};

bool supported(int n, int m, int d, int prec, int nlab);
size_t bytes(int n, int m, int d, int prec, int nlab, bool self);
// Lays the problem out inside buf (bytes() of it) and encodes its tensor maps.
cudaError_t layout(Problem& p, char* buf);
// Operands, squared norms, initial potentials and the biases of the first step, at the eps of rec[i][0]; the first
// records of every problem (count[i] of them, kTableSteps at most).
cudaError_t stage(Problem* const* p, const StepRec* const* rec, const int* count, int cnt, cudaStream_t st);
// Replaces the records.
cudaError_t upload(Problem* const* p, const StepRec* const* rec, const int* count, int cnt, cudaStream_t st);
// Steps [t0, t1) (counted since stage()) of cnt <= kMaxProblems problems of one kernel in lockstep, in one launch; the table's
// first record is that of step t_table. early: nothing happens once the problem has converged.
cudaError_t steps(Problem* const* p, int cnt, int t0, int t1, int t_table, bool early, double threshold, cudaStream_t st);
// Whether problems can share a launch.
bool lockstep(const Problem* const* p, int cnt);
// Stages the biases again for a step at eps: steps that an early stop skipped have left those of their own.
cudaError_t rebias(const Problem& p, double eps, cudaStream_t st);
// out[c] = potential + squared-norm shift for both clouds (null pointers are skipped).
cudaError_t emit(Problem* const* p, float* const (*out)[2], int cnt, cudaStream_t st);

// Kernel of these sizes: 1 operands resident, 2 streamed in K chunks, 3 / 4 the same by tiles of 256 x 256 / 128 x 128.
int kernel_of(int n, int m, int d, int prec, int nlab);
// Two-sided steps that problems have taken on the current device (-1: error).
long long two_sided_steps();

// Clocks that the CTAs of a solve wait for one another before they give up, for solves that the calling
// thread launches; returns what it was. Negative: the usual ~4 s.
long long set_meeting_limit(long long clocks);
int read_error_flag();
int clear_error_flag();

}  // namespace sym
}  // namespace fs
