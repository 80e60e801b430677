// Symmetric Sinkhorn steps with ONE exponential (and one contraction) per score entry for BOTH potentials.
//
// A Jacobi step updates f from the old g and g from the old f. With the shifted potentials f_hat, g_hat (cost
// C = cs|x-y|^2, logit scale 2cs/eps) both soft-mins are sums of the same numbers
//     E_ij = a_i b_j exp((f_hat_i + g_hat_j + 2cs x_i.y_j) / eps):
//     f_cand_i = f_hat_i + eps (log a_i - log sum_j E_ij),   g_cand_j = g_hat_j + eps (log b_j - log sum_i E_ij),
// so a tile of E serves the rows AND the columns. Both potentials ride in the contraction (three TF32 pieces each,
// exact to 2^-33): the row operand carries (x | 1 1 1 | f pieces), the column operand (y | g pieces | 1 1 1), and
// the drained accumulator times the logit scale is the finished exponent - no running maximum, no rescaling.
// A self-transport problem (x = y, a = b) has a symmetric E: only the tiles on one side of the diagonal are
// evaluated, their column sums standing in for the mirrored rows. (Coordinates are staged as scaled fp16 where that
// takes fewer K steps, see Layout; the scales are powers of two and are taken out of the logit scale again.)
//
// Which steps. Without a running maximum the sums must stay inside the fp32 exponent range. The end of a
// step knows, per row, L_i = log2 sum_j b_j 2^{z_ij} (z = the exponent without the weights) and the
// move dlt_i of its potential in log2 units (columns alike), and for the next step at eps' = eps / r, r >= 1:
//     log2 sum_j b_j 2^{r (z_ij + dlt_i + dlt_j)} <= r (L_i + dlt_i + max dlt_j) + (r - 1) max(-log2 b)
//                                                 >= r (L_i + dlt_i + min dlt_j) - (r - 1) max(0, log2 sum b)
// (upper: b_j 2^{z_ij} <= 2^{L_i}; lower: Jensen). A step is "two-sided" when these bounds keep every weighted row
// and column sum inside [2^-90, 2^120]; otherwise - the first steps of a solve from zero potentials at small eps,
// weights of zero, any NaN, points with scales of their own (wide_range) - the same kernel runs it "one-sided": rows of
// x, then rows of y, per-tile maxima, as (offset, sum) pairs. The decision is taken on the device from the same words by
// every CTA; the host enqueues the same launches either way. Simulated over eps from 0.0002 d to annealed schedules: two-sided
// from the second to the seventh step on, the row sums then within 2^+-30 of their weights.
//
// Launches. All steps of a solve (all that the same problems take) are ONE cooperative launch: per step the CTAs stream
// their runs of tiles, meet, turn the partial sums of their share of the points into potentials and biases, and meet again
// (end_step). What each step does comes from a table that is staged with the operands. With a second kernel per step
// for the finish, 4,096 points a side took 36 us per step, of which 13 were spent between the two kernels.
//
// Kernel layout (sym_kernel). Item = (128 streamed rows) x (256 stationary columns); the items of all problems
// of a launch, column tile after column tile, are cut into equal contiguous ranges, one per CTA, one CTA per SM.
// Holding the COLUMNS lets a thread (one TMEM lane = one row of each streamed tile) keep its 64 column sums in
// registers over a whole run of tiles: a column costs one FADD per entry and one cross-lane reduction per run.
// The row sum of a tile is one value per thread; warp 2 adds the four warpgroups' parts and stores one value per
// row and 256 columns (n*m/64 bytes in all, L2-resident at 50k x 50k), which the end of the step adds up.
//   warp 0 TMA producer, warp 1 tcgen05.mma issuer (M = 128, N = 256) and TMEM owner, warp 2 plan of the step and row-sum
//   collector, warps 4..19 four soft-max warpgroups, one per 64 columns.
// What bounds it: the ex2 pipe (16 per clock and SM): 2048 clocks per tile against 128 per K step of tensor pipe;
// operand traffic is one 128-row tile per 2048 clocks (10 bytes per clock and SM at d = 64 in fp16). A tile takes 2430
// clocks; a loop of the same loads, arithmetic, MMAs and barriers on its own takes 2400, without the barriers 2240. With
// 96 registers per soft-max thread instead of 112 it took 2790 (20 spilled words per tile).
// Measured on one B200 (debiased loss and gradient, d = 64, 100 steps, TF32 mode), against two soft-mins per step (first),
// two-sided steps of two launches (second):
// 50,000 x 50,000 307 -> 174 -> 160 ms (a step of the three problems 1.41 ms), 4,096 x 4,096 10.8 -> 3.8 -> 2.7 ms (23 us a
// step, 9 of them exponentials). 16,384 x 16,384 x 2,048, 50 steps: 201 -> 58 ms.
//
// Every mbarrier wait is bounded; on expiry the CTA raises an abort flag, lets its copies and MMAs land, frees its
// TMEM and returns, and a device-global error word records the event.
#include "fs_sym.cuh"
#include "fs_ptx.cuh"

#include <cudaTypedefs.h>

#include <algorithm>
#include <cstring>

namespace fs {
void count_launches(int k);
namespace sym {

using namespace fs::tc;  // PTX wrappers (internal linkage) and the tensor-map encoder

__device__ int g_sym_error = 0;
__device__ unsigned long long g_sym_two_sided = 0;  // steps of problems that ran two-sided

namespace {

constexpr int kBN = 256;           // stationary columns of a tile
constexpr int kWG = 4;             // soft-max warpgroups (64 columns each)
constexpr int kFirst = 4;         // first soft-max warp
constexpr int kThreads = 32 * kFirst + 128 * kWG;
constexpr int kAug = 6;            // bias columns: three pieces of either potential against ones
constexpr int kMaxCtas = 160;      // CTAs of a launch (sizes the column partials)
constexpr uint32_t kChunk = (128 + kBN) * 128;  // a ring stage of the K-streamed variant
constexpr int kOverhead = 15 * 1024;  // service area (below), alignment
// Shared memory of sym_kernel: partial ring [2 slots][offset | sum][kWG][128] of the row sums, barriers, words of the step,
// from kOperands on the operands. Fixed places: the soft-max loop has no register to spare for addresses.
constexpr int kBars = 2 * 2 * kWG * 128 * 4, kWords = kBars + 256, kOperands = 13 * 1024;
constexpr int kBFull = 0, kBEmpty = 2, kSFull = 4, kSEmpty = 6, kRFull = 8, kREmpty = 10, kDrain = 12, kAFull = 13;

struct Sub {
  CUtensorMap a_full[2], a_tail[2], b_full[2], b_tail[2];  // [side]: side 1 streams y against x
  Geo geo;
  const StepRec* sched;
  float* pot[2];
  const float* logw[2];
  const float* sq[2];
  float* opA[2];
  float* opB[2];
  float* out[2];
  float* pre[2];
  float* snap[2];
  double inv2cs;
};
template <int NS>
struct Launch {
  int nsub, nfull, ntail, nstage;
  int nb;      // column tiles in shared memory: with two, the next run's is loaded ahead
  int hs;      // leading K steps that hold fp16 coordinates
  int two_ok;  // 0: every problem of this launch runs one-sided
  int kc, kp;
  int t0, t1, t_table;  // steps of this launch, step of the first record
  int early;            // leave everything alone once the problem has converged
  double threshold;
  long long meet_limit;  // clocks that a CTA waits for the others (grid_wait)
  Sub sub[NS];
};

// ------------------------------------------------------------------ device helpers
__device__ __forceinline__ unsigned enc(float v) {
  const unsigned b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float dec(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld8_wait(uint32_t (&r)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
               :
               : "memory");
}

// Words of a problem that do not change over a launch, in shared memory: 24 lanes that read 24 problems from the kernel
// parameters do so in turn (4 us per step against 1).
struct Fixed {
  const uint4* slots;    // State::slot
  const StepRec* sched;
  int self, units;       // units: pieces of 128 points (end_step)
  float wa, la, wb, lb;  // largest -log2 and log2 of the weights of x, of y
  float mass_a, mass_b;  // bounds on log2 of their sums, at least 0
  float unit;            // scale of the products (pair_scale); negative: points with scales of their own
};
__device__ __forceinline__ Fixed fixed_words(const Sub& u) {
  const Geo& g = u.geo;
  const uint4 c = *reinterpret_cast<const uint4*>(g.st->cst);
  Fixed f;
  f.slots = reinterpret_cast<const uint4*>(g.st->slot[0]);
  f.sched = u.sched;
  f.self = g.self;
  f.units = (g.n[0] + 127) / 128 + (g.self ? 0 : (g.n[1] + 127) / 128);
  f.wa = dec(c.x); f.la = dec(c.y); f.wb = dec(c.z); f.lb = dec(c.w);
  f.mass_a = fmaxf(0.f, log2f((float)g.n[0]) + f.la);
  f.mass_b = fmaxf(0.f, log2f((float)g.n[1]) + f.lb);
  f.unit = wide_range(g.scales) ? -1.f : pair_scale(g.scales.range);
  return f;
}
// Whether the step that reads `slot` may run two-sided, at r = eps of the step before over its own (bounds of the header
// comment; NaN and inf say no).
__device__ __forceinline__ bool two_sided(const Fixed& f, int slot, float r) {
  const uint4* words = f.slots + 2 * slot;
  const uint4 x = __ldcg(words), y = f.self ? x : __ldcg(words + 1);
  if (!(r >= 0.999999f) || !(f.wa < 1000.f) || !(f.wb < 1000.f)) return false;
  const float uf = dec(x.x), lf = -dec(x.y), df_max = dec(x.z), df_min = -dec(x.w);
  const float ug = dec(y.x), lg = -dec(y.y), dg_max = dec(y.z), dg_min = -dec(y.w);
  const float row_hi = r * (uf + dg_max) + (r - 1.f) * f.wb, row_lo = r * (lf + dg_min) - (r - 1.f) * f.mass_b;
  const float col_hi = r * (ug + df_max) + (r - 1.f) * f.wa, col_lo = r * (lg + df_min) - (r - 1.f) * f.mass_a;
  return row_hi + f.la <= 120.f && row_lo - f.wa >= -90.f && col_hi + f.lb <= 120.f && col_lo - f.wb >= -90.f;
}

// Items of a launch: problem after problem; two-sided: column tile after column tile, all its row tiles (from the
// diagonal on for a self problem); one-sided: side 0 that way, then side 1. Every column tile of a two-sided problem of
// sym_kernel starts with an empty item, its head: the end of a run (64 sums per thread over the lanes, a partial per column)
// takes a soft-max warp as long as 1.2 tiles, and equal ranges of items that count it are equal in time (4,096 points a
// side, three problems: the slowest CTA's share of a step 14.9 -> 12.3 us).
struct Plan {
  int item0[kMaxProblems + 1];
  unsigned two;  // bit per problem
  int ctas;      // CTAs that take part (no more than items)
  int w_begin, w_end;  // items of this CTA (none begins right after a head: it begins with the head then)
};
__device__ __forceinline__ int head_items(const Geo& g, bool two) { return two && !g.by_tile ? 1 : 0; }
__device__ __forceinline__ int diag_tiles(const Geo& g) { return g.bn / g.bm; }  // row tiles on the diagonal: 1 or 2
// Items of column tile ct of a self problem, and the items before it: column tiles go in pairs (p, last - p), whose
// lengths add up to the same number for every pair, so that short and long runs spread evenly over the CTAs.
__device__ __forceinline__ int self_len(const Geo& g, int ct) { return g.nrt[0] - diag_tiles(g) * ct + head_items(g, true); }
__device__ __forceinline__ int self_offset(const Geo& g, int ct) {
  const int last = g.nct[0] - 1, pair = self_len(g, 0) + self_len(g, last);
  return 2 * ct <= last ? ct * pair : (last - ct) * pair + self_len(g, last - ct);
}
__device__ __forceinline__ int self_items(const Geo& g) {
  const int last = g.nct[0] - 1, pair = self_len(g, 0) + self_len(g, last);
  return (g.nct[0] / 2) * pair + ((g.nct[0] & 1) ? self_len(g, last / 2) : 0);
}
__device__ int item_count(const Geo& g, bool two) {
  const int one = g.nct[1] * (g.nrt[0] + head_items(g, two));
  if (two) return g.self ? self_items(g) : one;
  return g.self ? one : one + g.nct[0] * g.nrt[1];
}
// (a * b) / c for a * b of up to 63 bits; one 32-bit division where the product fits.
__device__ __forceinline__ int mul_div(int a, int b, int c) {
  const unsigned long long p = (unsigned long long)(unsigned)a * (unsigned)b;
  return p >> 32 ? (int)(p / (unsigned)c) : (int)((unsigned)p / (unsigned)c);
}
__device__ __forceinline__ int cta_first(int total, int ctas, int c) { return mul_div(total, c, ctas); }
__device__ __forceinline__ int cta_of(int total, int ctas, int t) {
  int c = mul_div(t, ctas, total);
  while (c + 1 < ctas && cta_first(total, ctas, c + 1) <= t) ++c;
  while (c > 0 && cta_first(total, ctas, c) > t) --c;
  return c;
}

// A run of row tiles against one column tile.
struct Run {
  int sub, side, ct, rt, len;
  int two;
  int strip0;            // first item of the column tile behind its head
  int step;              // items that the run takes up: len, and the head where it begins with one
  float *row_s, *row_m;  // where the row sums of its first row go
  float* col;            // where the column sums go (of the first warp of the four that have 32 rows of a tile each)
  int pitch, diag;       // of col from warp to warp; row tiles on the diagonal of a self problem
};
// The run that begins with item w.
template <class L>
__device__ Run locate(const L& P, const Plan& pl, int w, int w_end) {
  Run s;
  s.sub = 0;
  while (pl.item0[s.sub + 1] <= w) ++s.sub;
  const Geo& g = P.sub[s.sub].geo;
  s.two = (pl.two >> s.sub) & 1u;
  s.side = 0;
  const int head = head_items(g, s.two);
  int k = w - pl.item0[s.sub], rows = g.nrt[0];  // rows: row tiles of the column tile
  if (s.two && g.self) {
    const int last = g.nct[0] - 1, pair = self_len(g, 0) + self_len(g, last), p = k / pair;
    k -= p * pair;
    s.ct = p;
    if (k >= self_len(g, p)) {
      k -= self_len(g, p);
      s.ct = last - p;
    }
    rows = self_len(g, s.ct) - head;
  } else {
    if (!s.two && k >= g.nct[1] * rows) {
      k -= g.nct[1] * rows;
      s.side = 1;
      rows = g.nrt[1];
    }
    s.ct = k / (rows + head);
    k -= s.ct * (rows + head);
  }
  s.strip0 = w - k + head;
  const int skip = k < head ? 1 : 0, done = k < head ? 0 : k - head;
  const int left = rows - done, room = w_end - w - skip;
  s.len = left < room ? left : room;
  s.step = s.len + skip;
  s.rt = done + (s.two && g.self ? diag_tiles(g) * s.ct : 0);
  s.diag = s.two && g.self ? diag_tiles(g) * (s.ct + 1) - s.rt : 0;
  const size_t row = (size_t)s.ct * g.pad[s.side] + (size_t)s.rt * g.bm;
  s.row_s = g.rp_s[s.side] + row;
  s.row_m = g.rp_m[s.side] + row;
  const int piece = w <= s.strip0 ? 0 : (int)blockIdx.x - cta_of(pl.item0[P.nsub], pl.ctas, s.strip0);
  s.pitch = g.pad[1];
  s.col = g.cp + (size_t)piece * 4 * s.pitch + s.ct * g.bn;
  return s;
}
// The runs of a CTA, listed whenever the plan changes; the rest of a longer list is found again each time. 24 problems of a few
// column tiles each are about one run per CTA and problem at the most; longer lists are shares of many short column tiles (few
// row tiles), whose items are found by a dozen instructions more. 64 bytes a run, in the service area beside 24 problems' words.
constexpr int kRuns = 24;
template <class L>
__device__ __forceinline__ Run run_at(const L& P, const Plan& pl, const Run* runs, int nth, int w) {
  return nth < kRuns ? runs[nth] : locate(P, pl, w, pl.w_end);
}

// Plan, runs and records of step t, by one whole warp. In the copies for the CTA, `ratio` has become the factor that makes
// scores exponents: scale2 over the scales of both clouds.
template <class L>
__device__ __forceinline__ void begin_step(const L& P, const Fixed* fixed, int t, Plan* pl, Run* runs, StepRec* recs, int lane) {
  bool two = false;
  if (lane < P.nsub) {
    const float4* rec = reinterpret_cast<const float4*>(fixed[lane].sched + (t - P.t_table));
    float4 r0 = __ldcg(rec);
    const float4 r1 = __ldcg(rec + 1);
    two = P.two_ok && two_sided(fixed[lane], t % 3, r0.z);
    float4* to = reinterpret_cast<float4*>(recs + lane);
    r0.z = r0.w / fixed[lane].unit;  // exact: a power of two
    to[0] = r0;
    to[1] = r1;
  }
  const unsigned mask = __ballot_sync(0xffffffffu, two);
  // Steps with the plan of the step before, as all are after the first few of a solve, leave it as it is.
  if (t > P.t0 && mask == pl->two) return;
  __syncwarp();
  int pre = lane < P.nsub ? item_count(P.sub[lane].geo, two) : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, pre, o);
    if (lane >= o) pre += v;
  }
  if (lane < P.nsub) pl->item0[lane + 1] = pre;
  const int total = __shfl_sync(0xffffffffu, pre, P.nsub - 1);
  const int ctas = total < (int)gridDim.x ? total : (int)gridDim.x;
  if (lane == 0) {
    pl->item0[0] = 0;
    pl->two = mask;
    pl->ctas = ctas;
  }
  __syncwarp();
  if (runs && lane < 2) {
    int cut = (int)blockIdx.x < ctas ? cta_first(total, ctas, blockIdx.x + lane) : 0;
    if (cut > 0 && cut < total) {
      const Run s = locate(P, *pl, cut, total);
      if (cut == s.strip0 && head_items(P.sub[s.sub].geo, s.two)) --cut;
    }
    *(lane ? &pl->w_end : &pl->w_begin) = cut;
  }
  __syncwarp();
  if (runs && lane == 0)
    for (int k = 0, w = pl->w_begin; k < kRuns && w < pl->w_end; ++k) {
      runs[k] = locate(P, *pl, w, pl->w_end);
      w += runs[k].step;
    }
}

// Sums v[0..63] over the 32 lanes of the warp; lane l ends up with the totals of entries 2l and 2l + 1.
__device__ __forceinline__ void warp_columns(float (&v)[64], int lane) {
#pragma unroll
  for (int half = 32; half >= 2; half >>= 1) {
    const bool up = (lane & (half >> 1)) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float keep = up ? v[i + half] : v[i], send = up ? v[i] : v[i + half];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, half >> 1);
    }
  }
}

// ------------------------------------------------------------------ end of a step
// Writes the bias of a point (potential and log-weight over the dot scale: bd) as three TF32 pieces into its
// operand row.
__device__ __forceinline__ void write_bias(float* at, double bd) {
  const float hi = to_tf32((float)bd);
  const float mid = to_tf32((float)(bd - (double)hi));
  at[0] = hi;
  at[1] = mid;
  at[2] = to_tf32((float)(bd - (double)hi - (double)mid));
}
// What a point brings into its own sum: its potential and log-weight. Both stay out of it when they would only take bits
// from the finished sum, whose exponent the candidate subtracts again: a potential far above the eps of the step (the first
// steps of a point far from the rest: |x|^2 / eps, while its scores are |x||y| / eps), where an exponent of 2^31 rounds
// to more than fp32's range. Up to 2^20 its rounding is below 2^-4, that of potentials which fp32 holds anyway. A weight
// of zero (log = -1e5) stays out by itself. Two-sided steps need both inside: they run one-sided otherwise.
__device__ __forceinline__ double own_logw(double lw) { return lw < -700.0 ? 0.0 : lw; }
__device__ __forceinline__ bool own_inside(double pot, double own, double eps) {
  return fabs(pot + own * eps) * 1.4426950408889634 <= 1048576.0 * eps;
}

// The grid meets, twice per step: once all partial sums are in memory, and once the potentials and biases of the next step
// are. Launches are cooperative, so every CTA is resident. False: some CTA has given up (one of its own waits, or here), and
// all leave. `met` counts the meetings of this launch; leave_grid() puts the word back for the next one.
constexpr long long kMeetingLimit = 1ll << 33;  // clocks, ~4 s: the longest step of a solve takes milliseconds
constexpr unsigned kGivenUp = 0x80000000u;
__device__ __forceinline__ void grid_arrive(State* st, volatile int* abort_flag) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (*abort_flag) atomicOr(&st->bar_count, kGivenUp); else atomicAdd(&st->bar_count, 1u);
  }
}
__device__ __forceinline__ bool grid_wait(State* st, unsigned& met, volatile int* abort_flag, long long limit) {
  ++met;
  if (threadIdx.x == 0) {
    const unsigned goal = met * gridDim.x;
    const long long t_begin = clock64();
    for (unsigned seen = 0;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&st->bar_count) : "memory");
      if (seen & kGivenUp) *abort_flag = 1;
      if (seen >= goal) break;
      if (clock64() - t_begin > limit) atomicOr(&st->bar_count, kGivenUp);
    }
  }
  __syncthreads();
  return *abort_flag == 0;
}
__device__ __forceinline__ void leave_grid(State* st) {
  if (atomicAdd(&st->bar_leave, 1u) + 1u == gridDim.x) {
    st->bar_count = 0u;
    st->bar_leave = 0u;
  }
}

// 128 points of one cloud of one problem and where their partial sums are.
struct Unit {
  int sub, c, i0, base;  // base: first unit of the problem
  bool two;
  int k_rows, count;     // partials from row sums; all
  const float *rows, *cols;
};
// Unit number `unit` of a step; `from` is one that is not behind it. sub == nsub: there is none.
template <class L>
__device__ __forceinline__ Unit unit_at(const L& P, const Plan& plan, const Fixed* fixed, const Unit& from, int unit) {
  Unit v = from;
  while (v.sub < P.nsub && unit - v.base >= fixed[v.sub].units) v.base += fixed[v.sub++].units;
  if (v.sub == P.nsub) return v;
  const Geo& g = P.sub[v.sub].geo;
  const int nb0 = (g.n[0] + 127) / 128, block = unit - v.base;
  v.c = block < nb0 ? 0 : 1;
  v.i0 = (block - (v.c ? nb0 : 0)) * 128;
  v.two = (plan.two >> v.sub) & 1u;
  v.k_rows = v.count = 0;
  if (!v.two) {
    v.count = g.nct[g.self ? 0 : 1 - v.c];
    v.rows = g.rp_m[v.c] + v.i0;
    v.cols = g.rp_s[v.c] + v.i0;
    return v;
  }
  const int ct = v.i0 / g.bn;
  size_t col0 = 0;
  if (v.c == 0) v.k_rows = g.self ? ct + 1 : g.nct[1];
  v.count = v.k_rows;
  if (v.c == 1 || g.self) {
    if (g.by_tile) {
      col0 = g.self ? diag_tiles(g) * (ct + 1) : 0;
      v.count += g.nrt[0] - (int)col0;
    } else {
      const int total = plan.item0[P.nsub];
      const int head = head_items(g, true), len = g.self ? self_len(g, ct) - head : g.nrt[0];
      const int at = plan.item0[v.sub] + (g.self ? self_offset(g, ct) : ct * (g.nrt[0] + head)) + head;
      v.count += 4 * (cta_of(total, plan.ctas, at + len - 1) - cta_of(total, plan.ctas, at) + 1);
    }
  }
  v.rows = g.rp_s[0] + v.i0;
  v.cols = g.cp + col0 * g.pad[1] + v.i0;
  return v;
}

// The end of step t: the grid meets, adds the partial sums, updates the potentials in place (rounded once from fp64), stages
// the biases of the next step, records the ranges that decide how it runs, and meets again. By the 16 soft-max warps
// (first_warp ..): 128 points per team of eight, whose warps share the partials of each point and whose first four turn the
// sums into potentials; red: 1024 floats per team. False: no further step in this launch.
// Bound by latency at small sizes (one round of loads and one of fp64 arithmetic between the meetings; what does not
// depend on other CTAs is found and fetched while they are waited for) and by loads in flight at large ones (at 50,000
// points a side a point has 200 partials). Measured at 4,096 points a side, three problems: 3.1 us between
// the meetings, which take 1.4 us each (7.4 and 2.3 with 32 points per team of four warps, everything looked up behind the
// meeting and two more reads of its word), and 36 us against 134 at 50,000.
// WORK false: warps that only meet.
constexpr int kTeamWarps = 8;
template <bool WORK, class L>
__device__ __forceinline__ bool end_step(const L& P, const Plan& plan, const Fixed* fixed, const StepRec* recs, int t,
                                         float* red, int first_warp, unsigned& met, volatile int* abort_flag) {
  State* meet = P.sub[0].geo.st;
  const int w16 = (int)(threadIdx.x >> 5) - first_warp, lane = threadIdx.x & 31, slot = t % 3;
  const int team = w16 / kTeamWarps, warp = w16 % kTeamWarps;
  float* rd = red + team * (kTeamWarps * 128);
  Unit v;
  int unit = team * (int)gridDim.x + (int)blockIdx.x;
  v.sub = !WORK || w16 < 0 ? P.nsub : 0;
  v.base = 0;
  // what a potential needs besides the sums, of the point of a thread of the team's first four warps
  float pot_i = 0.f, logw_i = 0.f, sq_i = 0.f, unit_i = 1.f, snap_i = 0.f;
  auto team_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(2 + team), "n"(kTeamWarps * 32) : "memory"); };
  auto look = [&]() {
    v = unit_at(P, plan, fixed, v, unit);
    if (v.sub == P.nsub || warp >= 4) return;
    const Sub& u = P.sub[v.sub];
    const int i = v.i0 + warp * 32 + lane;
    if (i >= u.geo.n[v.c]) return;
    pot_i = __ldcg(u.pot[v.c] + i);
    logw_i = __ldg(u.logw[v.c] + i);
    sq_i = __ldcg(u.sq[v.c] + i);
    unit_i = fixed[v.sub].unit;
    if (unit_i < 0.f) unit_i = bias_factor(u.geo.scales, true, v.c, i);
    const unsigned todo = recs[v.sub].todo;
    if ((todo & kCheck) && (todo >> 8)) snap_i = __ldcg(u.snap[v.c] + i);
  };
  grid_arrive(meet, abort_flag);
  if (WORK) look();
  if (!grid_wait(meet, met, abort_flag, P.meet_limit)) return false;
#pragma unroll 1
  while (WORK && v.sub < P.nsub) {
    const Sub& u = P.sub[v.sub];
    const Geo& g = u.geo;
    const StepRec& rec = recs[v.sub];
    const int c = v.c, i = v.i0 + warp * 32 + lane;
    auto fetch = [&](const float* at) { return __ldcg(reinterpret_cast<const float4*>(at + 4 * lane)); };
    if (v.two) {
      const size_t row_pitch = g.pad[0], col_pitch = g.pad[1];
      float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
      for (int k = warp; k < v.count; k += 8 * kTeamWarps) {
        float4 x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int at = k + kTeamWarps * e;
          x[e] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (at < v.count) x[e] = fetch(at < v.k_rows ? v.rows + at * row_pitch : v.cols + (at - v.k_rows) * col_pitch);
        }
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          s0.x += x[e].x; s0.y += x[e].y; s0.z += x[e].z; s0.w += x[e].w;
          s1.x += x[e + 1].x; s1.y += x[e + 1].y; s1.z += x[e + 1].z; s1.w += x[e + 1].w;
        }
      }
      *reinterpret_cast<float4*>(rd + warp * 128 + 4 * lane) = make_float4(s0.x + s1.x, s0.y + s1.y, s0.z + s1.z, s0.w + s1.w);
    } else {
      // (offset, sum) pairs. Warp w and warp w + 4 find the largest offset of the pairs k = w mod 4, warp w adds them in their
      // order, so that potentials do not depend on how many warps load.
      const size_t pitch = g.pad[c];
      float4 m = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY), s = make_float4(0.f, 0.f, 0.f, 0.f);
      auto larger = [](const float4& p, const float4& q) {
        return make_float4(fmaxf(p.x, q.x), fmaxf(p.y, q.y), fmaxf(p.z, q.z), fmaxf(p.w, q.w));
      };
      for (int k = warp; k < v.count; k += 8 * kTeamWarps) {
        float4 x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int at = k + kTeamWarps * e;
          x[e] = fetch(v.rows + (at < v.count ? at : k) * pitch);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) m = larger(m, x[e]);
      }
      float4* own = reinterpret_cast<float4*>(rd + warp * 128 + 4 * lane);
      *own = m;
      team_sync();
      if (warp < 4) {
        float4* sum = own + 128;  // of warp w + 4: read here by the thread that writes its sum there
        m = larger(m, *sum);
        *own = m;
        for (int k = warp; k < v.count; k += 16) {
          float4 x[4], o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int at = k + 4 * e;
            x[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            o[e] = m;
            if (at < v.count) {
              x[e] = fetch(v.cols + at * pitch);
              o[e] = fetch(v.rows + at * pitch);
            }
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s.x += x[e].x * ex2(o[e].x - m.x); s.y += x[e].y * ex2(o[e].y - m.y);
            s.z += x[e].z * ex2(o[e].z - m.z); s.w += x[e].w * ex2(o[e].w - m.w);
          }
        }
        *sum = s;
      }
    }
    team_sync();
    if (warp < 4) {
      const float* at_m = rd + warp * 32 + lane;
      const float* at_s = at_m + 512;
      float m = 0.f, s = 0.f;
      if (v.two) {
        s = ((at_m[0] + at_m[128]) + (at_m[256] + at_m[384])) + ((at_s[0] + at_s[128]) + (at_s[256] + at_s[384]));
      } else {
        m = fmaxf(fmaxf(at_m[0], at_m[128]), fmaxf(at_m[256], at_m[384]));
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (at_s[k * 128] != 0.f) s += at_s[k * 128] * ex2(at_m[k * 128] - m);
      }
      float st_u = -INFINITY, st_l = -INFINITY, st_dx = -INFINITY, st_dn = -INFINITY, move = 0.f;
      if (i < g.n[c]) {
        // log2 of the weighted sum with the point's own bias inside; the candidate takes that bias out again
        const float l2 = m + log2f(fmaxf(s, 1e-40f));
        const double eps = (double)rec.eps, eps_next = (double)rec.eps_next;
        const double old = (double)pot_i, lw = (double)logw_i, own = own_logw(lw);
        const bool inside = own_inside(old, own, eps);
        const float damp = rec.damp[c];
        const double cand =
            (double)damp * ((inside ? old : 0.0) + eps * ((inside ? own : 0.0) - (double)l2 * 0.69314718055994530942));
        double nv = (1.0 - (double)rec.w) * old + (double)rec.w * cand;
        if (damp < 1.f) nv -= (double)(rec.w * (1.f - damp)) * (double)sq_i;
        const float now = (float)nv;
        u.pot[c][i] = now;
        const size_t at = (size_t)i * P.kp + P.kc;
        const double to_unit = u.inv2cs * (double)unit_i;
        const bool inside_next = own_inside((double)now, own, eps_next);
        write_bias(u.opA[c] + at + 3, inside_next ? ((double)now + own * eps_next) * to_unit : 0.0);
        write_bias(u.opB[c] + at, ((double)now + lw * eps_next) * to_unit);
        const float big_l = (float)((double)l2 - own * 1.4426950408889634);
        const float dlt = (float)((double)now - old) * (kLog2e / rec.eps);  // for the bounds alone, whose margins are octaves
        st_u = big_l + dlt;
        st_l = -st_u;
        st_dx = dlt;
        st_dn = -dlt;
        // no bound: the next step runs one-sided
        if (!(fabsf(st_u) < 1e30f) || !(fabsf(dlt) < 1e30f) || !inside || !inside_next) st_u = INFINITY;
        if (rec.todo & (kEmitPre | kEmitOut)) {
          const float std = now + sq_i;
          for (int k = c; k <= (g.self ? 1 : c); ++k) {
            if ((rec.todo & kEmitPre) && u.pre[k]) u.pre[k][i] = std;
            if ((rec.todo & kEmitOut) && u.out[k]) u.out[k][i] = std;
          }
        }
        if (rec.todo & kCheck) {
          move = fabsf(now - snap_i);
          if (move != move) move = INFINITY;  // as `max(...) < threshold` has it
          u.snap[c][i] = now;
        }
      }
      // one value per warp and word: unsigned order is float order (NaN: see above)
      const unsigned e_u = __reduce_max_sync(0xffffffffu, enc(st_u)), e_l = __reduce_max_sync(0xffffffffu, enc(st_l)),
                     e_x = __reduce_max_sync(0xffffffffu, enc(st_dx)), e_n = __reduce_max_sync(0xffffffffu, enc(st_dn));
      if (lane < 4)
        atomicMax(&g.st->slot[(slot + 1) % 3][4 * c + lane], lane == 0 ? e_u : (lane == 1 ? e_l : (lane == 2 ? e_x : e_n)));
      if (rec.todo & kCheck) {
        const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(move));
        if (lane == 0 && top) atomicMax(&g.st->delta[(rec.todo >> 8) & 1u], top);
      }
      if (unit == v.base && warp == 0) {  // once per problem
        if (lane == 31) g.ctrl->iters_used += 1;
        if (lane == 30 && v.two) atomicAdd(&g_sym_two_sided, 1ull);
        if (lane == 29 && (rec.todo & kCheck)) g.st->delta[((rec.todo >> 8) + 1u) & 1u] = 0u;
        if (lane >= 8 && lane < 16) g.st->slot[(slot + 2) % 3][lane - 8] = 0u;
      }
    }
    unit += (16 / kTeamWarps) * (int)gridDim.x;
    look();
    if (v.sub < P.nsub) team_sync();  // before rd is written again
  }
  // Early stopping: one problem per launch. Read here: behind the second meeting warp 2 of this CTA may be writing the records
  // of the next step (begin_step) while other warps still decide, and they all have to take this step's word.
  const unsigned todo = recs[0].todo;
  const bool check = P.early && (todo & kCheck);
  if (t + 1 == P.t1 && !check) return false;
  grid_arrive(meet, abort_flag);
  if (!grid_wait(meet, met, abort_flag, P.meet_limit)) return false;
  const unsigned nth = todo >> 8;
  if (check && nth > 0u && (double)__uint_as_float(__ldcg(&meet->delta[nth & 1u])) < P.threshold) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      P.sub[0].geo.ctrl->converged = 1;
      for (int k = 0; k < 3; ++k) meet->slot[k][0] = enc(INFINITY);  // the ranges describe another step's potentials
    }
    return false;
  }
  return t + 1 < P.t1;
}

// ------------------------------------------------------------------ the streaming kernel
// Bounded wait without a clock: one register. The bound is a number of polls, each of which the hardware may suspend for a
// while: 0.1 s at the least.
__device__ __forceinline__ bool wait_polling(uint32_t bar, uint32_t parity, uint32_t abort_at) {
  if (mbar_try_wait(bar, parity)) return true;
  for (int polls = 1 << 22; polls; --polls) {
    if (mbar_try_wait(bar, parity)) return true;
    int gone;
    asm volatile("ld.volatile.shared.s32 %0, [%1];" : "=r"(gone) : "r"(abort_at) : "memory");
    if (gone) return false;
  }
  asm volatile("st.volatile.shared.s32 [%0], %1;" ::"r"(abort_at), "r"(1) : "memory");
  return false;
}

// A warp's share of a two-sided run of len row tiles, the first of them number jt of the CTA: one lane is one row of each
// tile, lane_addr its 64 columns in the first accumulator. The row sum of a tile goes to part_at (and its other slot), the
// sums of columns 2 lane, 2 lane + 1 over the warp's 32 rows of all tiles are returned. The abort flag says whether all
// waits ended. A function of its own: 64 sums, two buffers and the loop's own words fill the registers, and what the caller
// keeps would otherwise be spilled in the loop (20 instructions per tile).
__device__ __noinline__ float2 two_sided_run(uint32_t lane_addr, uint32_t bar0, uint32_t part_at, float scale, int len, int jt,
                                             int diag) {  // diag: first tiles that add nothing to the column sums
  const int lane = threadIdx.x & 31;
  const uint32_t abort_at = bar0 + (kWords - kBars) + 4;
  const u64 sc = pk(scale, scale);
  u64 acc[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) acc[i] = 0ull;
  auto wait_tile = [&](int j) -> bool {
    if (!__all_sync(0xffffffffu, wait_polling(bar0 + 8 * kSFull + 8 * (j & 1), (j >> 1) & 1, abort_at))) return false;
    tc_fence_after();
    return true;
  };
  uint32_t ra[8], rb[8];
  // the first scores of a tile load while the last ones of the tile before are worked on
  bool ok = wait_tile(jt);
  if (ok) tmem_ld8_nowait(lane_addr + (uint32_t)((jt & 1) * kBN), ra);
#pragma unroll 1
  for (; ok && len > 0; --len, ++jt) {
    const uint32_t src = lane_addr + (uint32_t)((jt & 1) * kBN);
    u64 rs = 0ull;
    auto eat = [&](const uint32_t (&r)[8], int c) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float z0, z1;
        upk(mul2(pk(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1])), sc), z0, z1);
        const u64 e = pk(ex2(z0), ex2(z1));
        acc[c * 4 + k] = add2(acc[c * 4 + k], e);
        rs = add2(rs, e);
      }
    };
#pragma unroll
    for (int c = 0; c < 6; c += 2) {
      tmem_ld8_wait(ra);
      tmem_ld8_nowait(src + (c + 1) * 8, rb);
      eat(ra, c);
      tmem_ld8_wait(rb);
      tmem_ld8_nowait(src + (c + 2) * 8, ra);
      eat(rb, c + 1);
    }
    tmem_ld8_wait(ra);
    tmem_ld8_nowait(src + 56, rb);
    eat(ra, 6);
    tmem_ld8_wait(rb);
    tc_fence_before();  // every TMEM load of this warp from the buffer has landed
    __syncwarp();
    if (lane == 0) mbar_arrive(bar0 + 8 * kSEmpty + 8 * (jt & 1));
    if (len > 1) {
      ok = wait_tile(jt + 1);
      if (ok) tmem_ld8_nowait(lane_addr + (uint32_t)(((jt + 1) & 1) * kBN), ra);
    }
    eat(rb, 7);
    float a0, a1;
    upk(rs, a0, a1);
    ok = __all_sync(0xffffffffu, wait_polling(bar0 + 8 * kREmpty + 8 * (jt & 1), ((jt >> 1) & 1) ^ 1, abort_at)) && ok;
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(part_at + (jt & 1) * (2 * kWG * 128 * 4)), "f"(a0 + a1) : "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(bar0 + 8 * kRFull + 8 * (jt & 1));
    if (diag > 0) {
      --diag;
#pragma unroll
      for (int k = 0; k < 32; ++k) acc[k] = 0ull;
    }
  }
  // Where a wait gave up, the first scores of the next tile may still be on their way into registers that are used for other
  // things from here on.
  tmem_ld8_wait(ra);
  float v[64];
#pragma unroll
  for (int k = 0; k < 32; ++k) upk(acc[k], v[2 * k], v[2 * k + 1]);
  warp_columns(v, lane);
  return make_float2(v[0], v[1]);
}

// KS: the operands do not stay: K chunks of both (32 words; the last one may be partial) share the ring.
template <int NS, bool KS>
__global__ void __launch_bounds__(kThreads, 1) sym_kernel(const __grid_constant__ Launch<NS> P) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  // resident: nfull blocks of 32 words (128-byte swizzle) and ntail of 8 (32-byte swizzle) per operand row
  const uint32_t b_bytes = KS ? 0 : P.nfull * (kBN * 128) + P.ntail * (kBN * 32);
  const uint32_t a_bytes = KS ? kChunk : P.nfull * (128 * 128) + P.ntail * (128 * 32);
  uint8_t* b_smem = base + kOperands;
  uint8_t* a_smem = b_smem + P.nb * b_bytes;
  float* part = (float*)base;
  const int A_FULL = kAFull, A_EMPTY = kAFull + P.nstage, B_FULL = kBFull, B_EMPTY = kBEmpty, S_FULL = kSFull,
            S_EMPTY = kSEmpty, R_FULL = kRFull, R_EMPTY = kREmpty, DRAIN = kDrain;
  uint32_t* tmem_slot = (uint32_t*)(base + kWords);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  StepRec* recs = (StepRec*)(base + kWords + 16);
  Fixed* fixed = (Fixed*)(recs + NS);
  Plan* plan = (Plan*)(fixed + NS);
  Run* runs = (Run*)(((uintptr_t)(plan + 1) + 15) & ~(uintptr_t)15);
  static_assert(sizeof(StepRec) % 16 == 0 && kWords + 16 + NS * (sizeof(StepRec) + sizeof(Fixed)) + sizeof(Plan) + 16 +
                                                     kRuns * sizeof(Run) <= kOperands, "service area");
  const uint32_t bar0 = smem_u32(base + kBars);
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
  if (P.early && P.sub[0].geo.ctrl->converged) return;
  if (tid < P.nsub) fixed[tid] = fixed_words(P.sub[tid]);

  if (tid == 0) {
    for (int s = 0; s < P.nstage; ++s) {
      mbar_init(bar(A_FULL + s), 1);
      mbar_init(bar(A_EMPTY + s), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(B_FULL + i), 1);
      mbar_init(bar(B_EMPTY + i), 1);
      mbar_init(bar(S_FULL + i), 1);
      mbar_init(bar(S_EMPTY + i), 4 * kWG);  // one arrive per soft-max warp
      mbar_init(bar(R_FULL + i), 4 * kWG);
      mbar_init(bar(R_EMPTY + i), 1);
    }
    mbar_init(bar(DRAIN), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Counts that every role keeps over the steps: tiles, runs, K chunks (with the ring slot of the next one and its phase: a
  // division per chunk by the length of the ring cost the streamed kernel a tenth of its rate), meetings of the grid.
  int jt = 0, seg = 0, chunk = 0, ring = 0;
  uint32_t ring_phase = 0;
  auto ring_next = [&]() {
    ++chunk;
    if (++ring == P.nstage) { ring = 0; ring_phase ^= 1; }
  };
  unsigned met = 0;
  // The service warps and the soft-max warps go through the steps in loops of their own: the latter take registers from the
  // former.
  if (warp < kFirst) {
    registers_down();
#pragma unroll 1
    for (int t = P.t0;; ++t) {
      if (warp == 0) fence_proxy_async();  // the biases were written by ordinary stores, which the meeting has made visible
      if (warp == 2) begin_step(P, fixed, t, plan, runs, recs, lane);
      __syncthreads();
      const int w_begin = plan->w_begin, w_end = plan->w_end;
      const bool has_work = w_begin < w_end;
      if (warp == 0) {
        // ===================== TMA producer =====================
        if (KS && lane == 0 && has_work) {
          bool ok = true;
#pragma unroll 1
          for (int w = w_begin, nth = 0; ok && w < w_end; ++nth) {
            const Run s = run_at(P, *plan, runs, nth, w);
            const Sub& u = P.sub[s.sub];
#pragma unroll 1
            for (int t = 0; ok && t < s.len; ++t)
#pragma unroll 1
              for (int kc = 0; kc < P.nfull; ++kc) {
                const uint32_t full = bar(A_FULL + ring);
                if (!(ok = mbar_wait(bar(A_EMPTY + ring), ring_phase ^ 1, abort_flag, 2000))) break;
                mbar_expect_tx(full, kChunk);
                const uint32_t dst = smem_u32(a_smem + ring * kChunk);
                tma_load_2d(dst, &u.a_full[s.side], kc * 32, (s.rt + t) * 128, full);
                tma_load_2d(dst + 128 * 128, &u.b_full[s.side], kc * 32, s.ct * kBN, full);
                ring_next();
              }
            w += s.step;
          }
          if (*abort_flag)  // let every copy issued land before the CTA goes away
            for (int j = (chunk > P.nstage ? chunk - P.nstage : 0); j < chunk; ++j)
              mbar_wait_quiet(bar(A_FULL + j % P.nstage), (j / P.nstage) & 1);
        }
        if (!KS && lane == 0 && has_work) {
          int& issued = jt;
          int pre = 0;
          bool ok = true;
          auto load_a = [&](const Run& s, int t) -> bool {
            const Sub& u = P.sub[s.sub];
            const int st = issued % P.nstage;
            if (!mbar_wait(bar(A_EMPTY + st), ((issued / P.nstage) & 1) ^ 1, abort_flag, 2000)) return false;
            mbar_expect_tx(bar(A_FULL + st), a_bytes);
            const uint32_t dst = smem_u32(a_smem + st * a_bytes);
            const int row0 = (s.rt + t) * 128;
            for (int kb = 0; kb < P.nfull; ++kb)
              tma_load_2d(dst + kb * (128 * 128), &u.a_full[s.side], kb * 32, row0, bar(A_FULL + st));
            for (int k = 0; k < P.ntail; ++k)
              tma_load_2d(dst + P.nfull * (128 * 128) + k * (128 * 32), &u.a_tail[s.side], P.nfull * 32 + k * 8, row0,
                          bar(A_FULL + st));
            ++issued;
            return true;
          };
          auto load_b = [&](const Run& s) -> bool {  // column tile of run `seg`
            const int sl = seg % P.nb;
            // the column tile that was there must have been read by its last MMA
            if (!mbar_wait(bar(B_EMPTY + sl), ((seg / P.nb) & 1) ^ 1, abort_flag, 2000)) return false;
            mbar_expect_tx(bar(B_FULL + sl), b_bytes);
            const Sub& u = P.sub[s.sub];
            const uint32_t dst = smem_u32(b_smem + sl * b_bytes);
            for (int kb = 0; kb < P.nfull; ++kb)
              tma_load_2d(dst + kb * (kBN * 128), &u.b_full[s.side], kb * 32, s.ct * kBN, bar(B_FULL + sl));
            for (int k = 0; k < P.ntail; ++k)
              tma_load_2d(dst + P.nfull * (kBN * 128) + k * (kBN * 32), &u.b_tail[s.side], P.nfull * 32 + k * 8, s.ct * kBN,
                          bar(B_FULL + sl));
            ++seg;
            return true;
          };
          Run s = runs[0];
          ok = load_b(s);
#pragma unroll 1
          for (int w = w_begin, nth = 1; ok; ++nth) {
#pragma unroll 1
            for (int t = pre; ok && t < s.len; ++t) ok = load_a(s, t);
            w += s.step;
            if (!ok || w >= w_end) break;
            s = run_at(P, *plan, runs, nth, w);
            pre = 0;
            if (P.nb > 1) {
              ok = load_b(s);
            } else {
              // The first row tiles of the next run do not need its column tile: they fill ring slots meanwhile (every
              // slot waited for holds a tile that the MMA warp consumes without that column tile).
              const int npre = s.len < P.nstage ? s.len : P.nstage;
#pragma unroll 1
              for (; ok && pre < npre; ++pre) ok = load_a(s, pre);
              if (ok) ok = load_b(s);
            }
          }
          if (*abort_flag) {  // let every copy issued land before the CTA goes away
            for (int j = (seg > P.nb ? seg - P.nb : 0); j < seg; ++j) mbar_wait_quiet(bar(B_FULL + j % P.nb), (j / P.nb) & 1);
            for (int j = (issued > P.nstage ? issued - P.nstage : 0); j < issued; ++j)
              mbar_wait_quiet(bar(A_FULL + j % P.nstage), (j / P.nstage) & 1);
          }
        }
      } else if (warp == 1) {
        // ===================== MMA issuer (all lanes in the loop, one elected lane issues) =====================
        constexpr uint32_t idesc = make_idesc(kBN), idesc_h = make_idesc_f16(kBN);
        auto vote = [&](bool v) { return __all_sync(0xffffffffu, v) != 0; };
        bool ok = true;
        if (KS) {
#pragma unroll 1
          for (int w = w_begin, nth = 0; ok && w < w_end; ++nth) {
            const Run s = run_at(P, *plan, runs, nth, w);
            w += s.step;
#pragma unroll 1
            for (int i = 0; ok && i < s.len; ++i, ++jt) {
              const int buf = jt & 1;
              if (!vote(mbar_wait(bar(S_EMPTY + buf), ((jt >> 1) & 1) ^ 1, abort_flag, 2000))) break;
              tc_fence_after();
              const uint32_t d_tmem = tmem_base + (uint32_t)(buf * kBN);
#pragma unroll 1
              for (int kc = 0; kc < P.nfull; ++kc) {
                if (!vote(mbar_wait(bar(A_FULL + ring), ring_phase, abort_flag, 2000))) { ok = false; break; }
                tc_fence_after();
                if (elect_one()) {
                  const uint32_t at = smem_u32(a_smem + ring * kChunk), al = desc_lo(at), bl = desc_lo(at + 128 * 128);
                  const int steps = kc + 1 < P.nfull ? 4 : P.ntail;
#pragma unroll 1
                  for (int ks = 0; ks < steps; ++ks)
                    umma_step(kc * 4 + ks < P.hs, d_tmem, pack_desc(al + 2 * ks, kDescHi128), pack_desc(bl + 2 * ks, kDescHi128),
                              idesc, idesc_h, (kc | ks) != 0);
                  umma_commit(bar(A_EMPTY + ring));
                  if (kc + 1 == P.nfull) umma_commit(bar(S_FULL + buf));
                }
                __syncwarp();
                ring_next();
              }
            }
          }
        }
#pragma unroll 1
        for (int w = w_begin, nth = 0; !KS && ok && w < w_end; ++seg, ++nth) {
          const Run s = run_at(P, *plan, runs, nth, w);
          const int sl = seg % P.nb;
          if (!vote(mbar_wait(bar(B_FULL + sl), (seg / P.nb) & 1, abort_flag, 2000))) break;
          tc_fence_after();
#pragma unroll 1
          for (int i = 0; i < s.len; ++i, ++jt) {
            const int st = jt % P.nstage, buf = jt & 1;
            if (!vote(mbar_wait(bar(A_FULL + st), (jt / P.nstage) & 1, abort_flag, 2000)) ||
                !vote(mbar_wait(bar(S_EMPTY + buf), ((jt >> 1) & 1) ^ 1, abort_flag, 2000))) {
              ok = false;
              break;
            }
            tc_fence_after();
            if (elect_one()) {
              const uint32_t d_tmem = tmem_base + (uint32_t)(buf * kBN);
              int left = P.hs;  // fp16 K steps to go
              uint32_t al = desc_lo(smem_u32(a_smem + st * a_bytes)), bl = desc_lo(smem_u32(b_smem + sl * b_bytes));
              uint32_t acc = 0;
#pragma unroll 1
              for (int kb = 0; kb < P.nfull; ++kb) {
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                  umma_step(left > ks, d_tmem, pack_desc(al + 2 * ks, kDescHi128), pack_desc(bl + 2 * ks, kDescHi128), idesc,
                            idesc_h, acc);
                  acc = 1;
                }
                left -= 4;
                al += (128 * 128) >> 4;
                bl += (kBN * 128) >> 4;
              }
#pragma unroll 1
              for (int k = 0; k < P.ntail; ++k) {
                umma_step(left > k, d_tmem, pack_desc(al, kDescHi32), pack_desc(bl, kDescHi32), idesc, idesc_h, acc);
                acc = 1;
                al += (128 * 32) >> 4;
                bl += (kBN * 32) >> 4;
              }
              umma_commit(bar(S_FULL + buf));
              umma_commit(bar(A_EMPTY + st));
            }
            __syncwarp();
          }
          if (elect_one()) umma_commit(bar(B_EMPTY + sl));  // the column tile may be replaced once these MMAs retired
          __syncwarp();
          w += s.step;
        }
        __syncwarp();
        if (*abort_flag && lane == 0) {  // wait (bounded) for every MMA issued before TMEM is freed
          umma_commit(bar(DRAIN));
          mbar_wait_quiet(bar(DRAIN), 0);
        }
      } else if (warp == 2) {
        // ===================== row-sum collector: adds the warpgroups' parts, one value per row =====================
        bool ok = true;
#pragma unroll 1
        for (int w = w_begin, nth = 0; ok && w < w_end; ++nth) {
          const Run s = run_at(P, *plan, runs, nth, w);
#pragma unroll 1
          for (int i = 0; i < s.len; ++i, ++jt) {
            const int slot = jt & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(bar(R_FULL + slot), (jt >> 1) & 1, abort_flag, 1000))) {
              ok = false;
              break;
            }
            const float *pm = part + slot * 2 * kWG * 128 + lane, *ps = pm + kWG * 128;
#pragma unroll 1
            for (int r = 0; r < 128; r += 32) {  // one row per lane at a time: this warp has few registers
              const size_t to = (size_t)i * 128 + r + lane;
              const float s0 = ps[r], s1 = ps[128 + r], s2 = ps[256 + r], s3 = ps[384 + r];
              if (s.two) {
                s.row_s[to] = (s0 + s1) + (s2 + s3);
              } else {
                const float m0 = pm[r], m1 = pm[128 + r], m2 = pm[256 + r], m3 = pm[384 + r];
                const float top = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
                s.row_m[to] = top;
                s.row_s[to] = (s0 * ex2(m0 - top) + s1 * ex2(m1 - top)) + (s2 * ex2(m2 - top) + s3 * ex2(m3 - top));
              }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(R_EMPTY + slot));
          }
          w += s.step;
        }
      }
      __syncwarp();
      if (!end_step<false>(P, *plan, fixed, recs, t, part, kFirst, met, abort_flag)) break;
    }
  } else {
    // ===================== soft-max warpgroups =====================
    registers_up();
#pragma unroll 1
    for (int t = P.t0;; ++t) {
      __syncthreads();
      const int w_begin = plan->w_begin, w_end = plan->w_end;
      const bool has_work = w_begin < w_end;
      const int wg = (warp - kFirst) >> 2, q = warp & 3;  // columns [64 wg, 64 wg + 64) of a tile; TMEM lane quarter
      const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + wg * 64;
      const int trow = q * 32 + lane;
      bool ok = true;
      auto wait_tile = [&](int j) -> bool {
        if (!mbar_wait(bar(S_FULL + (j & 1)), (j >> 1) & 1, abort_flag)) return false;
        __syncwarp();
        tc_fence_after();
        return true;
      };
      auto release_tile = [&]() {  // every TMEM load of this warp from the buffer has landed
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(S_EMPTY + (jt & 1)));
      };
      auto post = [&](float m, float s) -> bool {  // this thread's part of the row sum goes to the collector
        const int slot = jt & 1;
        if (!mbar_wait(bar(R_EMPTY + slot), ((jt >> 1) & 1) ^ 1, abort_flag)) return false;
        float* pp = part + slot * 2 * kWG * 128 + wg * 128 + trow;
        pp[0] = m;
        pp[kWG * 128] = s;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(R_FULL + slot));
        return true;
      };
#pragma unroll 1
      for (int w = w_begin, nth = 0; w < w_end; ++nth) {
        const Run s = run_at(P, *plan, runs, nth, w);
        const float pair = recs[s.sub].ratio;
        if (s.two) {
          float2 sums = make_float2(0.f, 0.f);
          if (ok) sums = two_sided_run(lane_addr, bar0, smem_u32(part + kWG * 128 + wg * 128 + trow), pair, s.len, jt, s.diag);
          jt += s.len;
          ok = __all_sync(0xffffffffu, *abort_flag == 0) != 0;
          if (ok) {  // one row of partials per warp (32 rows of each tile): no barrier at the end of a run
            float* to = s.col + (size_t)(q * s.pitch + wg * 64 + 2 * lane);
            *reinterpret_cast<float2*>(to) = sums;
          }
        } else {
          const Geo& g = P.sub[s.sub].geo;
          const bool wide = fixed[s.sub].unit < 0.f;
#pragma unroll 1
          for (int i = 0; ok && i < s.len; ++i, ++jt) {
            if (!(ok = wait_tile(jt))) break;
            const uint32_t src = lane_addr + (uint32_t)((jt & 1) * kBN);
            const float scale = wide ? recs[s.sub].scale2 * g.scales.inv[s.side][(s.rt + i) * 128 + trow] : pair;
            uint32_t r[32];
            float m_run = run_init(scale), off = __fmul_rn(scale, m_run), sum = 0.f;
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
              tmem_ld32_nowait(src + c * 32, r);
              tmem_ld_wait(r);
              if (wide) unscale_columns(r, g.scales.inv[1 - s.side] + s.ct * kBN + wg * 64 + c * 32);
              float cm = __uint_as_float(r[0]);
#pragma unroll
              for (int k = 1; k < 31; k += 2) cm = max3(cm, __uint_as_float(r[k]), __uint_as_float(r[k + 1]));
              m_run = fmaxf(m_run, fmaxf(cm, __uint_as_float(r[31])));
              // the rounded product is the offset all terms are relative to (must not be contracted into an FMA)
              const float off_new = __fmul_rn(scale, m_run);
              float s0 = sum * ex2(off - off_new), s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
              for (int k = 0; k < 32; k += 4) {
                s0 += ex2(fmaf(__uint_as_float(r[k]), scale, -off_new));
                s1 += ex2(fmaf(__uint_as_float(r[k + 1]), scale, -off_new));
                s2 += ex2(fmaf(__uint_as_float(r[k + 2]), scale, -off_new));
                s3 += ex2(fmaf(__uint_as_float(r[k + 3]), scale, -off_new));
              }
              sum = (s0 + s1) + (s2 + s3);
              off = off_new;
            }
            release_tile();
            if (!(ok = post(off, sum))) break;
          }
        }
        w += s.step;
      }
      __syncwarp();
      if (!end_step<true>(P, *plan, fixed, recs, t, part, kFirst, met, abort_flag)) break;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
  if (tid == 0) {
    leave_grid(P.sub[0].geo.st);
    if (*abort_flag) atomicExch(&g_sym_error, 1);
  }
}

// ------------------------------------------------------------------ long contractions
// Tiles of 128*NHALF rows x BN columns whose operands stream through the ring in K chunks; the tensor pipe (or the
// operand traffic) binds, so the epilogue may spend shuffles on the column sums: one value per column and tile.
//   256 x 256, one accumulator per half: 64 operand bytes per clock at full tensor rate; the epilogue is exposed
//   128 x 128, two accumulators: for problems with too few 256 x 256 tiles to go round
// Items go to the CTAs in turn, in groups of kGroup column tiles, so that the tiles in flight share their operands.
// warp 0 producer, warps 1 and 3 MMA issuers of a half, warps 4.. PARTS warpgroups per half.
constexpr int kGroup = 12;

template <int NHALF, int BN, int NBUF, int PARTS>
__global__ void __launch_bounds__(128 + 128 * NHALF * PARTS, 1) sym_wide_kernel(const __grid_constant__ Launch<1> P) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  constexpr int BM = 128 * NHALF, NSYNC = BM * PARTS, GROUPS = 4 * NHALF;
  constexpr uint32_t kAHalf = 128 * 128, kStage = NHALF * kAHalf + BN * 128;
  constexpr uint32_t kTmemCols = NHALF * NBUF * BN;
  constexpr int CH = BN / 32 / PARTS;  // 32-column chunks of a tile owned by a warpgroup
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* colred = (float*)(base + P.nstage * kStage);   // [2][GROUPS][BN] column sums of 32 rows each
  float* rowred = colred + 2 * GROUPS * BN;             // [2][offset | sum][PARTS][BM]
  uint64_t* bars = (uint64_t*)(rowred + 2 * 2 * PARTS * BM);
  const int FULL = 0, EMPTY = P.nstage, S_FULL = 2 * P.nstage, S_EMPTY = S_FULL + NHALF * NBUF,
            DRAIN = S_EMPTY + NHALF * NBUF, NBARS = DRAIN + 2;
  StepRec* recs = (StepRec*)(bars + ((NBARS + 1) & ~1));
  Fixed* fixed = (Fixed*)(recs + 1);
  uint32_t* tmem_slot = (uint32_t*)(fixed + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  Plan* plan = (Plan*)(tmem_slot + 2);
  auto bar = [&](int i) { return smem_u32(bars + i); };
  const Sub& u = P.sub[0];
  const Geo& g = u.geo;
  if (P.early && g.ctrl->converged) return;
  if (tid == 0) *fixed = fixed_words(u);

  if (tid == 0) {
    for (int s = 0; s < P.nstage; ++s) {
      mbar_init(bar(FULL + s), 1);
      mbar_init(bar(EMPTY + s), NHALF);
    }
    for (int i = 0; i < NHALF * NBUF; ++i) {
      mbar_init(bar(S_FULL + i), 1);
      mbar_init(bar(S_EMPTY + i), 4 * PARTS);
    }
    mbar_init(bar(DRAIN), 1);
    mbar_init(bar(DRAIN + 1), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Counts that every role keeps over the steps: tiles, K chunks, meetings of the grid.
  int jt = 0, chunk = 0;
  unsigned met = 0;
#pragma unroll 1
  for (int t = P.t0;; ++t) {
    if (warp == 0) fence_proxy_async();  // the biases were written by ordinary stores, which the meeting has made visible
    if (warp == 2) begin_step(P, fixed, t, plan, nullptr, recs, lane);
    __syncthreads();
    const int total = plan->item0[1];
    const bool two = plan->two & 1u;
    // Item k: (side, row tile, column tile).
    auto locate_tile = [&](int k, int& side, int& rt, int& ct) {
      side = 0;
      if (two && g.self) {
        const Run s = locate(P, *plan, k, k + 1);
        rt = s.rt;
        ct = s.ct;
        return;
      }
      if (k >= g.nct[1] * g.nrt[0]) {
        k -= g.nct[1] * g.nrt[0];
        side = 1;
      }
      const int rows = g.nrt[side], cols = g.nct[1 - side], grp = k / (kGroup * rows), c0 = grp * kGroup;
      const int width = cols - c0 < kGroup ? cols - c0 : kGroup, in = k - grp * kGroup * rows;
      rt = in / width;
      ct = c0 + in - rt * width;
    };

    if (warp == 0) {
      if (lane == 0) {
        int& issued = chunk;
        bool ok = true;
#pragma unroll 1
        for (int k = blockIdx.x; ok && k < total; k += gridDim.x) {
          int side, rt, ct;
          locate_tile(k, side, rt, ct);
#pragma unroll 1
          for (int kc = 0; kc < P.nfull; ++kc) {
            const int s = issued % P.nstage;
            if (!mbar_wait(bar(EMPTY + s), ((issued / P.nstage) & 1) ^ 1, abort_flag, 2000)) { ok = false; break; }
            mbar_expect_tx(bar(FULL + s), kStage);
            const uint32_t dst = smem_u32(base + (size_t)s * kStage);
#pragma unroll
            for (int h = 0; h < NHALF; ++h)
              tma_load_2d(dst + h * kAHalf, &u.a_full[side], kc * 32, rt * BM + h * 128, bar(FULL + s));
            tma_load_2d(dst + NHALF * kAHalf, &u.b_full[side], kc * 32, ct * BN, bar(FULL + s));
            ++issued;
          }
        }
        if (*abort_flag)  // let every copy issued land before the CTA goes away
          for (int j = (issued > P.nstage ? issued - P.nstage : 0); j < issued; ++j)
            mbar_wait_quiet(bar(FULL + j % P.nstage), (j / P.nstage) & 1);
      }
    } else if (warp == 1 || (warp == 3 && NHALF == 2)) {
      const int h = warp == 1 ? 0 : 1;
      constexpr uint32_t idesc = make_idesc(BN), idesc_h = make_idesc_f16(BN);
      auto vote = [&](bool v) { return __all_sync(0xffffffffu, v) != 0; };
      bool ok = true;
      int s = chunk % P.nstage;
      uint32_t ph = (chunk / P.nstage) & 1;
#pragma unroll 1
      for (int k = blockIdx.x; ok && k < total; k += gridDim.x, ++jt) {
        const int buf = h * NBUF + jt % NBUF;
        if (!vote(mbar_wait(bar(S_EMPTY + buf), ((jt / NBUF) & 1) ^ 1, abort_flag, 2000))) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * BN);
#pragma unroll 1
        for (int kc = 0; kc < P.nfull; ++kc) {
          if (!vote(mbar_wait(bar(FULL + s), ph, abort_flag, 2000))) { ok = false; break; }
          tc_fence_after();
          const uint32_t at = smem_u32(base + (size_t)s * kStage);
          const uint32_t al = desc_lo(at + h * kAHalf), bl = desc_lo(at + NHALF * kAHalf);
          const int steps = kc + 1 < P.nfull ? 4 : P.ntail;
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            if (ks < steps && elect_one())
              umma_step(kc * 4 + ks < P.hs, d_tmem, pack_desc(al + 2 * ks, kDescHi128), pack_desc(bl + 2 * ks, kDescHi128),
                        idesc, idesc_h, (kc | ks) != 0);
          if (elect_one()) umma_commit(bar(EMPTY + s));
          __syncwarp();
          if (++s == P.nstage) { s = 0; ph ^= 1; }
        }
        chunk += P.nfull;
        if (!ok) break;
        if (elect_one()) umma_commit(bar(S_FULL + buf));
        __syncwarp();
      }
      __syncwarp();
      if (*abort_flag && lane == 0) {
        umma_commit(bar(DRAIN + h));
        mbar_wait_quiet(bar(DRAIN + h), 0);
      }
    } else if (warp >= 4) {
      const int wg = (warp - 4) >> 2, h = wg / PARTS, part = wg % PARTS, q = warp & 3;
      const int trow = h * 128 + q * 32 + lane, et = tid - 128;  // row inside the tile, epilogue thread
      const float pair = recs[0].ratio;
      const bool wide = fixed->unit < 0.f;
      bool ok = true;
#pragma unroll 1
      for (int k = blockIdx.x; k < total; k += gridDim.x, ++jt) {  // also after an abort: every warp takes every barrier
        int side, rt, ct;
        locate_tile(k, side, rt, ct);
        const int buf = h * NBUF + jt % NBUF, sl = jt & 1;
        if (ok) ok = mbar_wait(bar(S_FULL + buf), (jt / NBUF) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok) != 0;
        const float scale = wide ? recs[0].scale2 * g.scales.inv[side][rt * BM + trow] : pair;
        float m_run = run_init(scale), off = two ? 0.f : __fmul_rn(scale, m_run), sum = 0.f;
        if (ok) {
          tc_fence_after();
          const uint32_t src = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN) + part * CH * 32;
#pragma unroll 1
          for (int c = 0; c < CH; ++c) {
            uint32_t r[32];
            tmem_ld32_nowait(src + c * 32, r);
            tmem_ld_wait(r);
            if (c == CH - 1) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(bar(S_EMPTY + buf));
            }
            if (wide) unscale_columns(r, g.scales.inv[1 - side] + ct * BN + (part * CH + c) * 32);
            float v[32], s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
            if (two) {
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                s0 += v[i] = ex2(__uint_as_float(r[i]) * scale);
                s1 += v[i + 1] = ex2(__uint_as_float(r[i + 1]) * scale);
                s2 += v[i + 2] = ex2(__uint_as_float(r[i + 2]) * scale);
                s3 += v[i + 3] = ex2(__uint_as_float(r[i + 3]) * scale);
              }
              sum += (s0 + s1) + (s2 + s3);
#pragma unroll
              for (int half = 16; half >= 1; half >>= 1) {  // over the warp's rows; lane l keeps column l
                const bool up = (lane & half) != 0;
#pragma unroll
                for (int i = 0; i < half; ++i) {
                  const float keep = up ? v[i + half] : v[i], send = up ? v[i] : v[i + half];
                  v[i] = keep + __shfl_xor_sync(0xffffffffu, send, half);
                }
              }
              colred[(sl * GROUPS + h * 4 + q) * BN + (part * CH + c) * 32 + lane] = v[0];
            } else {
              float cm = __uint_as_float(r[0]);
#pragma unroll
              for (int i = 1; i < 31; i += 2) cm = max3(cm, __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
              m_run = fmaxf(m_run, fmaxf(cm, __uint_as_float(r[31])));
              const float off_new = __fmul_rn(scale, m_run);
              s0 = sum * ex2(off - off_new);
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                s0 += ex2(fmaf(__uint_as_float(r[i]), scale, -off_new));
                s1 += ex2(fmaf(__uint_as_float(r[i + 1]), scale, -off_new));
                s2 += ex2(fmaf(__uint_as_float(r[i + 2]), scale, -off_new));
                s3 += ex2(fmaf(__uint_as_float(r[i + 3]), scale, -off_new));
              }
              sum = (s0 + s1) + (s2 + s3);
              off = off_new;
            }
          }
          float* rr = rowred + (sl * 2 * PARTS + part) * BM + trow;
          rr[0] = off;
          rr[PARTS * BM] = sum;
        }
        // one barrier per tile: the buffers alternate, and a thread reaches the barrier of tile j + 1 only after it
        // has read those of tile j
        asm volatile("bar.sync 1, %0;" ::"n"(NSYNC) : "memory");
        if (ok) {
          if (et < BM) {
            const float* rm = rowred + sl * 2 * PARTS * BM + et;
            const float* rs = rm + PARTS * BM;
            const size_t at = (size_t)ct * g.pad[side] + (size_t)rt * BM + et;
            float m = rm[0], s = 0.f;
            if (two) {
#pragma unroll
              for (int i = 0; i < PARTS; ++i) s += rs[i * BM];
              g.rp_s[0][at] = s;
            } else {
#pragma unroll
              for (int i = 1; i < PARTS; ++i) m = fmaxf(m, rm[i * BM]);
#pragma unroll
              for (int i = 0; i < PARTS; ++i) s += rs[i * BM] * ex2(rm[i * BM] - m);
              g.rp_m[side][at] = m;
              g.rp_s[side][at] = s;
            }
          }
          const int col = et - (NSYNC - BN);  // the other end of the threads
          if (two && col >= 0) {
            const float* cr = colred + sl * GROUPS * BN + col;
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < GROUPS; ++i) s += cr[i * BN];
            g.cp[(size_t)rt * g.pad[1] + ct * BN + col] = s;
          }
        }
      }
    }

    __syncwarp();
    if (!end_step<true>(P, *plan, fixed, recs, t, rowred, 4, met, abort_flag)) break;
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  if (tid == 0) {
    leave_grid(g.st);
    if (*abort_flag) atomicExch(&g_sym_error, 1);
  }
}

// ------------------------------------------------------------------ staging
struct StageSub {
  const float* src[2];
  const float* logw[2];
  const float* init[2];
  const int* label[2];
  const float* W;
  int V;
  float w_coef, cs_sq;
  double eps, inv2cs;
  int n[2], pad[2], self;
  float* opA[2];
  float* opB[2];
  float* pot[2];
  float* sq[2];
  float* inv[2];
  OperandScales scales;
  State* st;
  Ctrl* ctrl;
};
template <int NS>
struct StageLaunch {
  int nsub, d, kcoord, kc, kp, hs, prec, cloud;
  StageSub sub[NS];
};

// Step records of up to kMaxProblems problems, one block each; with `fresh` the control words of a solve too.
template <int NR>
struct Upload {
  int fresh;
  struct Job {
    StepRec* to;
    State* st;
    Ctrl* ctrl;
    int from, count;
  } job[kMaxProblems];
  StepRec rec[NR];
};
template <int NR>
__global__ void sym_upload_kernel(const __grid_constant__ Upload<NR> P) {
  const typename Upload<NR>::Job& j = P.job[blockIdx.x];
  for (int k = threadIdx.x; k < j.count; k += blockDim.x) j.to[k] = P.rec[j.from + k];
  if (threadIdx.x || !P.fresh) return;
  State* st = j.st;
  for (int k = 0; k < 8; ++k) {
    st->slot[0][k] = enc(INFINITY);  // nothing is known about the first step: it runs one-sided
    st->slot[1][k] = st->slot[2][k] = 0u;
  }
  for (int k = 0; k < 4; ++k) st->cst[k] = 0u;
  for (int k = 0; k < kRangeWords; ++k) st->range[k] = 0u;
  st->delta[0] = st->delta[1] = 0u;
  st->bar_count = st->bar_leave = 0u;
  j.ctrl->delta_bits = 0u; j.ctrl->converged = 0; j.ctrl->have_prev = 0; j.ctrl->iters_used = 0;
}

template <int NS>
__global__ void __launch_bounds__(256) sym_range_kernel(const __grid_constant__ StageLaunch<NS> P) {
  const StageSub& u = P.sub[blockIdx.y];
  const int c = blockIdx.z;  // a self problem reads its cloud twice: both ranges are its own
  row_ranges(u.src[c], u.n[c], u.pad[c], P.d, blockIdx.x, gridDim.x, c == 1 && u.self ? nullptr : u.inv[c], u.st->range, c,
             2 * gridDim.x, scale_octaves(P.prec));
}

// One warp per point of cloud P.cloud: both operand rows (stage_coord, label columns), the squared
// norm, the initial shifted potential and the biases of the first step; column layout as in the header comment with
// kc = coordinate and label columns.
template <int NS>
__global__ void __launch_bounds__(256) sym_stage_kernel(const __grid_constant__ StageLaunch<NS> P) {
  __shared__ unsigned wmax[2];
  const StageSub& u = P.sub[blockIdx.y];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = P.cloud;
  if ((c == 1 && u.self) || (int)blockIdx.x >= u.pad[c] / 8) return;
  if (threadIdx.x < 2) wmax[threadIdx.x] = 0u;
  __syncthreads();
  const int r = (int)blockIdx.x * 8 + warp;
  const bool real = r < u.n[c];
  const int d = P.d, kc = P.kc, kp = P.kp, kcoord = P.kcoord;
  const bool wide = wide_range(u.scales);
  const float own = coord_factor(u.scales, wide, c, r), ones = ones_factor(u.scales, wide, c, r),
              unit = bias_factor(u.scales, wide, c, r);
  const float* src = u.src[c] + (size_t)r * d;
  float* rowA = u.opA[c] + (size_t)r * kp;
  float* rowB = u.opB[c] + (size_t)r * kp;
  float nrm = 0.f;
  if (real)
    for (int k = lane; k < d; k += 32) { const float v = src[k]; nrm = fmaf(v, v, nrm); }
#pragma unroll
  for (int o = 16; o; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
  const int lab = (real && u.V > 0) ? u.label[c][r] : 0;
  for (int k = lane; k < kp; k += 32) {
    if (k >= kc && k < kc + 6) continue;
    float va = 0.f, vb = 0.f;
    if (k < kcoord && real) {
      stage_coord(src, k, d, P.prec == 0 ? 1 : 3, P.hs, own, va, vb);
    } else if (k < kc && real) {
      const int v = (k - kcoord) / 3, piece = (k - kcoord) % 3;
      va = lab == v ? ones : 0.f;
      // column role: the table entry between every class v of the other cloud and this point's label
      const float w = unit * u.w_coef * u.W[c == 0 ? lab * u.V + v : v * u.V + lab];
      const float h = to_tf32(w), mid = to_tf32(w - h), low = to_tf32(w - h - mid);
      vb = piece == 0 ? h : (piece == 1 ? mid : low);
    }
    rowA[k] = va;
    rowB[k] = vb;
  }
  if (lane < 3) {
    rowA[kc + lane] = ones;
    rowB[kc + 3 + lane] = ones;
  }
  if (lane == 0) {
    if (real) {
      const float sq = u.cs_sq * nrm;
      const float pot = (u.init[c] ? u.init[c][r] : 0.f) - sq;
      const float lw = u.logw[c][r];
      u.sq[c][r] = sq;
      u.pot[c][r] = pot;
      const double in = own_logw(lw);
      write_bias(rowA + kc + 3, own_inside((double)pot, in, u.eps) ? ((double)pot + in * u.eps) * u.inv2cs * (double)unit : 0.0);
      write_bias(rowB + kc, ((double)pot + (double)lw * u.eps) * u.inv2cs * (double)unit);
      float l2 = lw * kLog2e;
      if (!(fabsf(l2) < 1e30f) || wide) l2 = -1e30f;  // such a weight keeps every step one-sided, as a wide range does
      atomicMax(&wmax[0], enc(-l2));
      atomicMax(&wmax[1], enc(l2));
    } else {  // padded points contribute 2^(-2^100 * scale) = 0 in either role
      rowA[kc + 3] = kMaskBias; rowA[kc + 4] = 0.f; rowA[kc + 5] = 0.f;
      rowB[kc] = kMaskBias; rowB[kc + 1] = 0.f; rowB[kc + 2] = 0.f;
    }
  }
  __syncthreads();
  if (threadIdx.x < 2 && wmax[threadIdx.x] != 0u) {
    atomicMax(&u.st->cst[2 * c + threadIdx.x], wmax[threadIdx.x]);
    if (u.self) atomicMax(&u.st->cst[2 + threadIdx.x], wmax[threadIdx.x]);
  }
}

// Stages the biases again for a step at eps (eps_next), from the potentials as they are. One thread per point.
struct Rebias {
  Geo geo;
  const float* pot[2];
  const float* logw[2];
  float* opA[2];
  float* opB[2];
  double eps_next, inv2cs;
  int kp, kc;
};
__global__ void sym_rebias_kernel(const __grid_constant__ Rebias P) {
  const Rebias& u = P;
  const Geo& g = P.geo;
  const int c = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n[c]) return;
  const double pot = (double)u.pot[c][i], lw = (double)u.logw[c][i], own = own_logw(lw);
  const double to_unit = u.inv2cs * (double)bias_factor(g.scales, wide_range(g.scales), c, i);
  const size_t at = (size_t)i * P.kp + P.kc;
  write_bias(u.opA[c] + at + 3, own_inside(pot, own, u.eps_next) ? (pot + own * u.eps_next) * to_unit : 0.0);
  write_bias(u.opB[c] + at, (pot + lw * u.eps_next) * to_unit);
}

struct EmitJobs {
  struct Job {
    const float *pot[2], *sq[2];
    float* out[2];
    int n[2];
  } job[kMaxProblems];
};
__global__ void sym_emit_kernel(const __grid_constant__ EmitJobs P) {
  const EmitJobs::Job& j = P.job[blockIdx.y];
  const int c = blockIdx.z, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < j.n[c] && j.out[c]) j.out[c][i] = j.pot[c][i] + j.sq[c][i];
}

// ------------------------------------------------------------------ host side
thread_local long long t_meeting_limit = kMeetingLimit;  // of the solves that this thread launches, no other's
enum Kind { RESIDENT = 0, STREAMED = 1, WIDE = 2, SMALL = 3 };
struct Shape {
  int kind, bm, bn;
  int nb, hs, kc, kp, nfull, ntail, nstage;  // K-streamed kinds: nfull chunks of 32 words, the last one with ntail K steps
  size_t smem;
};

inline int tiles(int n, int t) { return (n + t - 1) / t; }

Shape plan_shape(int n, int m, int d, int prec, int nlab) {
  Shape s{};
  const tc::Layout l = tc::operand_layout(d, prec, nlab, kAug);
  s.kc = l.kc;
  s.kp = l.kp;
  s.hs = l.hs;
  const size_t row = (size_t)s.kp * 4, budget = kSmemMax - kOverhead;
  s.bm = 128;
  s.bn = kBN;
  if ((kBN + 2 * 128) * row <= budget) {  // 256 columns and two row tiles fit
    s.kind = RESIDENT;
    s.nfull = s.kp / 32;
    s.ntail = (s.kp % 32) / 8;
    s.nb = (2 * kBN + 3 * 128) * row <= budget ? 2 : 1;
    s.nstage = (int)((budget - s.nb * kBN * row) / (128 * row));
    if (s.nstage > 4) s.nstage = 4;
    s.smem = s.nb * kBN * row + s.nstage * 128 * row + kOverhead;
    if (s.smem < (size_t)kSmemMin) s.smem = kSmemMin;
    return s;
  }
  s.nfull = tiles(s.kp, 32);
  s.ntail = (s.kp - (s.nfull - 1) * 32) / 8;
  // Clocks of a whole pass: rounds of the SMs times the clocks of a tile. Operand chunks arrive at about 45 bytes
  // per clock and SM (48, 64, 32 KB per chunk for the three shapes) next to the epilogue, which only the single
  // accumulator of the 256 x 256 tile exposes.
  const long long nk = s.nfull;
  auto rounds = [&](int bm, int bn) { return ((long long)tiles(n, bm) * tiles(m, bn) + 147) / 148; };
  auto most = [](long long a, long long b) { return a > b ? a : b; };
  const long long mid = rounds(128, 256) * most(1090 * nk, 2200) + 2200, wide = rounds(256, 256) * (1400 * nk + 8000),
                  little = rounds(128, 128) * most(720 * nk, 2200) + 2200;
  if (mid <= wide && mid <= little) {
    s.kind = STREAMED;
    s.nstage = 4;
    s.smem = s.nstage * (size_t)kChunk + kOverhead;
    return s;
  }
  s.kind = little < wide ? SMALL : WIDE;
  s.bm = s.bn = s.kind == SMALL ? 128 : 256;
  s.nstage = s.kind == SMALL ? 6 : 3;
  s.smem = s.nstage * (size_t)(2 * s.bm * 128) + 28 * 1024;
  return s;
}

// Rows of the column-partial buffer: CTAs that can share one column tile (twice the even share for the triangular
// item list of a self problem, plus the two ends), never more than there are row tiles.
int max_pieces(int n, int m) {
  const long long share = 2ll * kMaxCtas / tiles(m, kBN) + 2;
  return (int)(share < tiles(n, 128) ? share : tiles(n, 128));
}

// The scratch of the per-tile row sums grows with n*m (16 bytes per 256 entries and side): up to this much.
constexpr size_t kMaxPartialBytes = size_t(2) << 30;

size_t carve(Problem& p, char* buf) {
  Carve c{buf};
  const Shape sh = plan_shape(p.n[0], p.n[1], p.d, p.prec, 3 * p.lab.V);
  p.kc = sh.kc;
  p.kp = sh.kp;
  p.kind = sh.kind;
  Geo& g = p.geo;
  g = Geo{};
  g.self = p.self ? 1 : 0;
  g.bm = sh.bm;
  g.bn = sh.bn;
  g.by_tile = sh.kind >= WIDE ? 1 : 0;
  for (int k = 0; k < 2; ++k) {
    g.n[k] = p.n[k];
    g.pad[k] = tc::detail::pad256(p.n[k]);
    g.nrt[k] = tiles(p.n[k], sh.bm);
    g.nct[k] = tiles(p.n[k], sh.bn);
  }
  p.ctrl = c.take<Ctrl>(1);
  g.ctrl = p.ctrl;
  g.st = c.take<State>(1);
  p.sched = p.table = c.take<StepRec>(kTableSteps);
  float* inv[2];
  inv[0] = c.take<float>(g.pad[0]);
  inv[1] = p.self ? inv[0] : c.take<float>(g.pad[1]);
  if (sh.hs && g.st) {
    g.scales.range = g.st->range;
    for (int k = 0; k < 2; ++k) g.scales.inv[k] = inv[k];
  }
  for (int k = 0; k < 2; ++k) {
    if (k == 1 && p.self) {
      p.opA[1] = p.opA[0]; p.opB[1] = p.opB[0]; p.pot[1] = p.pot[0]; p.sq[1] = p.sq[0];
      g.rp_m[1] = g.rp_m[0]; g.rp_s[1] = g.rp_s[0];
      break;
    }
    p.opA[k] = c.take<float>((size_t)g.pad[k] * p.kp);
    p.opB[k] = c.take<float>((size_t)g.pad[k] * p.kp);
    p.pot[k] = c.take<float>(g.pad[k]);
    p.sq[k] = c.take<float>(g.pad[k]);
    g.rp_m[k] = c.take<float>((size_t)g.nct[1 - k] * g.pad[k]);
    g.rp_s[k] = c.take<float>((size_t)g.nct[1 - k] * g.pad[k]);
  }
  g.cp = c.take<float>((size_t)(g.by_tile ? g.nrt[0] : 4 * max_pieces(p.n[0], p.n[1])) * g.pad[1]);
  return c.off;
}

template <int NS>
cudaError_t steps_n(Problem* const* p, int cnt, int t0, int t1, int t_table, bool early, double threshold, cudaStream_t st) {
  const Problem& p0 = *p[0];
  const Shape sh = plan_shape(p0.n[0], p0.n[1], p0.d, p0.prec, 3 * p0.lab.V);
  Launch<NS> lp;
  lp.nsub = cnt;
  lp.nfull = sh.nfull; lp.ntail = sh.ntail; lp.nstage = sh.nstage;
  lp.hs = sh.hs;
  lp.nb = sh.nb;
  lp.kc = sh.kc; lp.kp = sh.kp;
  lp.t0 = t0; lp.t1 = t1; lp.t_table = t_table;
  lp.early = early ? 1 : 0;
  lp.threshold = threshold;
  lp.meet_limit = t_meeting_limit;
  long long most = 0;
  for (int i = 0; i < cnt; ++i) {
    const Problem& q = *p[i];
    Sub& u = lp.sub[i];
    u.geo = q.geo;
    u.sched = q.sched;
    u.inv2cs = 0.5 / (double)q.cs_dot;
    for (int k = 0; k < 2; ++k) {
      u.a_full[k] = q.map[4 * k]; u.a_tail[k] = q.map[4 * k + 1];
      u.b_full[k] = q.map[4 * k + 2]; u.b_tail[k] = q.map[4 * k + 3];
      u.pot[k] = q.pot[k]; u.logw[k] = q.logw[k]; u.sq[k] = q.sq[k]; u.opA[k] = q.opA[k]; u.opB[k] = q.opB[k];
      u.out[k] = q.out[k]; u.pre[k] = q.pre[k]; u.snap[k] = q.snap[k];
    }
    most += (long long)q.geo.nct[1] * q.geo.nrt[0] + (q.self ? 0 : (long long)q.geo.nct[0] * q.geo.nrt[1]);
  }
  int ctas = tc::detail::free_ctas();
  if (ctas > kMaxCtas) ctas = kMaxCtas;
  // With a CTA for every one-sided item there is nothing to share: both sides run next to each other on SMs that
  // would idle, without the column reduction and without a bound on the range.
  lp.two_ok = most > ctas;
  if (most < ctas) ctas = (int)most;
  auto go = [&](auto kern, int threads) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;  // the CTAs meet twice per step
    at[0].val.cooperative = 1;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = sh.smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    // fewer CTAs where this context may not use every SM
    for (int grid = ctas;; grid = (grid + 1) / 2) {
      cfg.gridDim = dim3(grid);
      e = cudaLaunchKernelEx(&cfg, kern, lp);
      if (e != cudaErrorCooperativeLaunchTooLarge || grid == 1) return e;
      (void)cudaGetLastError();
    }
  };
  cudaError_t e = cudaErrorInvalidValue;
  if (sh.kind == RESIDENT) e = go(sym_kernel<NS, false>, kThreads);
  if (sh.kind == STREAMED) e = go(sym_kernel<NS, true>, kThreads);
  if constexpr (NS == 1) {
    if (sh.kind == WIDE) e = go(sym_wide_kernel<2, 256, 1, 2>, 128 + 512);
    if (sh.kind == SMALL) e = go(sym_wide_kernel<1, 128, 2, 4>, 128 + 512);
  }
  count_launches(1);
  return e;
}

// Fills and launches one block of records; from[i] < 0: nothing for problem i.
template <int NR>
cudaError_t upload_n(Problem* const* p, const StepRec* const* rec, const int* from, const int* count, int cnt, bool fresh,
                     cudaStream_t st) {
  Upload<NR> u;
  u.fresh = fresh ? 1 : 0;
  for (int i = 0; i < cnt; ++i) {
    u.job[i].to = p[i]->table;
    u.job[i].st = p[i]->geo.st;
    u.job[i].ctrl = p[i]->ctrl;
    u.job[i].from = from[i] < 0 ? 0 : from[i];
    u.job[i].count = from[i] < 0 ? 0 : count[i];
    if (from[i] >= 0) std::copy(rec[i], rec[i] + count[i], u.rec + from[i]);
  }
  sym_upload_kernel<NR><<<cnt, 64, 0, st>>>(u);
  count_launches(1);
  return cudaGetLastError();
}

// Records of all problems in as few launches as they fit; problems with equal records share the first one's table.
cudaError_t upload_all(Problem* const* p, const StepRec* const* rec, const int* count, int cnt, bool fresh, cudaStream_t st) {
  constexpr int kSmall = 64, kMost = 900;  // records of a launch (kernel parameters stay under 32 KB)
  int from[kMaxProblems], room = 0;
  cudaError_t e = cudaSuccess;
  auto flush = [&]() {
    if (e == cudaSuccess)
      e = room <= kSmall ? upload_n<kSmall>(p, rec, from, count, cnt, fresh, st) : upload_n<kMost>(p, rec, from, count, cnt, fresh, st);
    fresh = false;
    room = 0;
  };
  for (int i = 0; i < cnt; ++i) from[i] = -1;
  for (int i = 0; i < cnt; ++i) {
    int same = 0;
    while (same < i && !(count[same] == count[i] && std::memcmp(rec[same], rec[i], count[i] * sizeof(StepRec)) == 0)) ++same;
    p[i]->sched = p[same]->table;
    if (same < i) continue;
    if (room + count[i] > kMost) {
      flush();
      for (int k = 0; k < i; ++k) from[k] = -1;
    }
    from[i] = room;
    room += count[i];
  }
  flush();
  return e;
}

template <int NS>
cudaError_t stage_n(Problem* const* p, const StepRec* const* rec, const int* count, int cnt, cudaStream_t st) {
  StageLaunch<NS> lp;
  lp.nsub = cnt; lp.d = p[0]->d; lp.prec = p[0]->prec;
  const tc::Layout lay = tc::operand_layout(lp.d, lp.prec, 3 * p[0]->lab.V, kAug);
  lp.kcoord = lay.kcoord; lp.kc = lay.kc; lp.kp = lay.kp; lp.hs = lay.hs;
  int blocks[2] = {0, 0};  // one launch per cloud; problems of one cloud only have no second one
  for (int i = 0; i < cnt; ++i) {
    const Problem& q = *p[i];
    StageSub& u = lp.sub[i];
    for (int k = 0; k < 2; ++k) {
      u.src[k] = q.src[k]; u.logw[k] = q.logw[k]; u.init[k] = q.init[k]; u.label[k] = q.lab.lab[k];
      u.n[k] = q.n[k]; u.pad[k] = q.geo.pad[k];
      u.opA[k] = q.opA[k]; u.opB[k] = q.opB[k]; u.pot[k] = q.pot[k]; u.sq[k] = q.sq[k];
      u.inv[k] = const_cast<float*>(q.geo.scales.inv[k]);
    }
    u.scales = q.geo.scales;
    u.W = q.lab.W; u.V = q.lab.V; u.w_coef = -q.lab.lam_w / (2.0f * q.cs_dot);
    u.cs_sq = q.cs_sq; u.eps = rec[i][0].eps; u.inv2cs = 0.5 / (double)q.cs_dot;
    u.self = q.self ? 1 : 0; u.st = q.geo.st; u.ctrl = q.ctrl;
    blocks[0] = q.geo.pad[0] / 8 > blocks[0] ? q.geo.pad[0] / 8 : blocks[0];
    if (!q.self) blocks[1] = q.geo.pad[1] / 8 > blocks[1] ? q.geo.pad[1] / 8 : blocks[1];
  }
  const cudaError_t e = upload_all(p, rec, count, cnt, true, st);
  if (e != cudaSuccess) return e;
  if (lp.hs) {  // both scales are known before anything is staged
    const int pad = 8 * (blocks[0] > blocks[1] ? blocks[0] : blocks[1]);
    sym_range_kernel<NS><<<dim3(tc::detail::range_blocks(pad, lp.d), cnt, 2), 256, 0, st>>>(lp);
    count_launches(1);
  }
  for (lp.cloud = 0; lp.cloud < 2; ++lp.cloud)
    if (blocks[lp.cloud]) {
      sym_stage_kernel<NS><<<dim3(blocks[lp.cloud], cnt), 256, 0, st>>>(lp);
      count_launches(1);
    }
  return cudaGetLastError();
}

}  // namespace

bool supported(int n, int m, int d, int prec, int nlab) {
  if ((prec != 0 && prec != 1) || n <= 0 || m <= 0 || d <= 0) return false;
  // items are numbered with 32-bit integers; the partials must fit their budget
  const Shape sh = plan_shape(n, m, d, prec, nlab);
  const size_t rows = (size_t)tiles(m, sh.bn) * tc::detail::pad256(n) + (size_t)tiles(n, sh.bn) * tc::detail::pad256(m);
  return 2 * rows * sizeof(float) <= kMaxPartialBytes;
}

size_t bytes(int n, int m, int d, int prec, int nlab, bool self) {
  Problem p;
  p.self = self;
  p.n[0] = n; p.n[1] = m; p.d = d; p.prec = prec; p.lab.V = nlab / 3;
  return carve(p, nullptr) + 1024;
}

cudaError_t layout(Problem& p, char* buf) {
  carve(p, (char*)(((uintptr_t)buf + 1023) & ~(uintptr_t)1023));
  const Shape sh = plan_shape(p.n[0], p.n[1], p.d, p.prec, 3 * p.lab.V);
  const bool wide_box = sh.kind != RESIDENT || sh.nfull > 0;  // 32-word blocks exist (of a short row: only tails)
  const CUtensorMapSwizzle full = wide_box ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_32B;
  bool ok = true;
  for (int k = 0; k < 2 && ok; ++k) {
    const int o = 1 - k;  // the column operand of side k belongs to the other cloud
    ok &= tc::detail::encode_map(&p.map[4 * k], p.opA[k], p.geo.pad[k], sh.kp, wide_box ? 32 : 8, 128, full);
    ok &= tc::detail::encode_map(&p.map[4 * k + 1], p.opA[k], p.geo.pad[k], sh.kp, 8, 128, CU_TENSOR_MAP_SWIZZLE_32B);
    ok &= tc::detail::encode_map(&p.map[4 * k + 2], p.opB[o], p.geo.pad[o], sh.kp, wide_box ? 32 : 8, sh.bn, full);
    ok &= tc::detail::encode_map(&p.map[4 * k + 3], p.opB[o], p.geo.pad[o], sh.kp, 8, sh.bn, CU_TENSOR_MAP_SWIZZLE_32B);
  }
  return ok ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t stage(Problem* const* p, const StepRec* const* rec, const int* count, int cnt, cudaStream_t st) {
  if (cnt < 1 || cnt > kMaxProblems) return cudaErrorInvalidValue;
  if (cnt == 1) return stage_n<1>(p, rec, count, cnt, st);
  if (cnt <= 3) return stage_n<3>(p, rec, count, cnt, st);
  return stage_n<kMaxProblems>(p, rec, count, cnt, st);
}

cudaError_t upload(Problem* const* p, const StepRec* const* rec, const int* count, int cnt, cudaStream_t st) {
  return upload_all(p, rec, count, cnt, false, st);
}

bool lockstep(const Problem* const* p, int cnt) {
  for (int i = 0; i < cnt; ++i)
    if (p[i]->kind >= WIDE || p[i]->kind != p[0]->kind) return cnt == 1;
  return true;
}

cudaError_t steps(Problem* const* p, int cnt, int t0, int t1, int t_table, bool early, double threshold, cudaStream_t st) {
  if (cnt < 1 || cnt > kMaxProblems || t1 <= t0 || !lockstep(p, cnt)) return cudaErrorInvalidValue;
  if (cnt == 1) return steps_n<1>(p, cnt, t0, t1, t_table, early, threshold, st);
  if (cnt <= 3) return steps_n<3>(p, cnt, t0, t1, t_table, early, threshold, st);
  return steps_n<kMaxProblems>(p, cnt, t0, t1, t_table, early, threshold, st);
}

cudaError_t rebias(const Problem& p, double eps, cudaStream_t st) {
  Rebias f;
  f.kc = p.kc; f.kp = p.kp;
  f.geo = p.geo;
  for (int k = 0; k < 2; ++k) {
    f.pot[k] = p.pot[k]; f.logw[k] = p.logw[k]; f.opA[k] = p.opA[k]; f.opB[k] = p.opB[k];
  }
  f.eps_next = (float)eps;
  f.inv2cs = 0.5 / (double)p.cs_dot;
  const int rows = p.n[0] > p.n[1] ? p.n[0] : p.n[1];
  sym_rebias_kernel<<<dim3((rows + 255) / 256, p.self ? 1 : 2), 256, 0, st>>>(f);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t emit(Problem* const* p, float* const (*out)[2], int cnt, cudaStream_t st) {
  EmitJobs jobs;
  int rows = 1;
  for (int i = 0; i < cnt; ++i)
    for (int k = 0; k < 2; ++k) {
      EmitJobs::Job& j = jobs.job[i];
      j.pot[k] = p[i]->pot[k]; j.sq[k] = p[i]->sq[k]; j.out[k] = out[i][k]; j.n[k] = p[i]->n[k];
      rows = p[i]->n[k] > rows ? p[i]->n[k] : rows;
    }
  count_launches(1);
  sym_emit_kernel<<<dim3((rows + 255) / 256, cnt, 2), 256, 0, st>>>(jobs);
  return cudaGetLastError();
}

int kernel_of(int n, int m, int d, int prec, int nlab) {
  const int kind = plan_shape(n, m, d, prec, nlab).kind;
  return kind == RESIDENT ? 1 : (kind == STREAMED ? 2 : (kind == WIDE ? 3 : 4));
}

long long two_sided_steps() {
  unsigned long long v = 0;
  return cudaMemcpyFromSymbol(&v, g_sym_two_sided, sizeof(v)) == cudaSuccess ? (long long)v : -1;
}

long long set_meeting_limit(long long clocks) {
  const long long was = t_meeting_limit;
  t_meeting_limit = clocks < 0 ? kMeetingLimit : clocks;
  return was;
}

int read_error_flag() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_sym_error, sizeof(int)) != cudaSuccess) return -1;
  return v ? 1 : 0;
}
int clear_error_flag() {
  const int zero = 0;
  return cudaMemcpyToSymbol(g_sym_error, &zero, sizeof(int)) == cudaSuccess ? 0 : -1;
}

}  // namespace sym
}  // namespace fs
