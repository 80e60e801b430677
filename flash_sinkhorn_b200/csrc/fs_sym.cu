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
// Which steps. Without a running maximum the sums must stay inside the fp32 exponent range. After every step the
// finalising kernel knows, per row, L_i = log2 sum_j b_j 2^{z_ij} (z = the exponent without the weights) and the
// move dlt_i of its potential in log2 units (columns alike), and for the next step at eps' = eps / r, r >= 1:
//     log2 sum_j b_j 2^{r (z_ij + dlt_i + dlt_j)} <= r (L_i + dlt_i + max dlt_j) + (r - 1) max(-log2 b)
//                                                 >= r (L_i + dlt_i + min dlt_j) - (r - 1) max(0, log2 sum b)
// (upper: b_j 2^{z_ij} <= 2^{L_i}; lower: Jensen). A step is "two-sided" when these bounds keep every weighted row
// and column sum inside [2^-90, 2^120]; otherwise - the first steps of a solve from zero potentials at small eps,
// weights of zero, any NaN, points with scales of their own (wide_range) - the same kernel runs it "one-sided": rows of
// x, then rows of y, per-tile maxima, as (offset, sum) pairs. The decision is taken on the device from the same words by every CTA; the host enqueues the
// same launches either way. Simulated over eps from 0.0002 d to annealed schedules: two-sided from the second to
// the seventh step on, the row sums then within 2^+-30 of their weights.
//
// Kernel layout (sym_kernel). Item = (128 streamed rows) x (256 stationary columns); the items of all problems
// of a launch, column tile after column tile, are cut into equal contiguous ranges, one per CTA, one CTA per SM.
// Holding the COLUMNS lets a thread (one TMEM lane = one row of each streamed tile) keep its 64 column sums in
// registers over a whole run of tiles: a column costs one FADD per entry and one cross-lane reduction per run.
// The row sum of a tile is one value per thread; warp 2 adds the four warpgroups' parts and stores one value per
// row and 256 columns (n*m/64 bytes in all, L2-resident at 50k x 50k), which the finalising kernel adds up.
//   warp 0 TMA producer, warp 1 tcgen05.mma issuer (M = 128, N = 256) and TMEM owner, warp 2 row-sum
//   collector, warps 4..19 four soft-max warpgroups, one per 64 columns.
// What bounds it: the ex2 pipe (16 per clock and SM): 2048 clocks per tile against 128 per K step of tensor pipe;
// operand traffic is one 128-row tile per 2048 clocks (10 bytes per clock and SM at d = 64 in fp16).
// Measured on one B200 (debiased loss and gradient, d = 64, 100 steps, TF32 mode), against two soft-mins per step:
// 50,000 x 50,000 307 -> 172 ms (a two-sided step of the three problems 1.45 ms, 12 exponentials per clock and SM, the
// ex2 pipe 78 % busy), 4,096 x 4,096 10.8 -> 3.8 ms (36 us a step, 9 of them exponentials: the chain of the two
// launches binds). 16,384 x 16,384 x 2,048, 50 steps: 201 -> 58 ms.
//
// Every mbarrier wait is bounded; on expiry the CTA raises an abort flag, lets its copies and MMAs land, frees its
// TMEM and returns, and a device-global error word records the event.
#include "fs_sym.cuh"
#include "fs_ptx.cuh"

#include <cudaTypedefs.h>

namespace fs {
void count_launches(int k);
namespace sym {

using namespace fs::tc;  // PTX wrappers (internal linkage) and the tensor-map encoder

__device__ int g_sym_error = 0;
__device__ unsigned long long g_sym_two_sided = 0;  // steps of problems that ran two-sided

namespace {

constexpr int kBN = 256;           // stationary columns of a tile
constexpr int kWG = 4;             // soft-max warpgroups (64 columns each)
constexpr int kThreads = 128 + 128 * kWG;
constexpr int kAug = 6;            // bias columns: three pieces of either potential against ones
constexpr int kMaxCtas = 160;      // CTAs of a launch (sizes the column partials)
constexpr uint32_t kChunk = (128 + kBN) * 128;  // a ring stage of the K-streamed variant
constexpr int kOverhead = 15 * 1024;  // barriers, plan, partial ring, column reduction, alignment

struct Sub {
  CUtensorMap a_full[2], a_tail[2], b_full[2], b_tail[2];  // [side]: side 1 streams y against x
  Geo geo;
  float scale2;  // 2*cs*log2e/eps
};
template <int NS>
struct Launch {
  int nsub, nfull, ntail, nstage, slot;
  int nb;      // column tiles in shared memory: with two, the next run's is loaded ahead
  int hs;      // leading K steps that hold fp16 coordinates
  int two_ok;  // 0: every problem of this launch runs one-sided
  Sub sub[NS];
};
struct FinSub {
  Geo geo;
  float* pot[2];
  const float* logw[2];
  const float* sq[2];
  float* opA[2];
  float* opB[2];
  double eps, eps_next, inv2cs, log2e_eps;
  float w, damp[2], shiftcoef[2];
};
template <int NS>
struct FinLaunch {
  int nsub, kc, kp, slot, ctas, two_ok;
  FinSub sub[NS];
};

// ------------------------------------------------------------------ device helpers
__device__ __forceinline__ unsigned enc(float v) {
  const unsigned b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float dec(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

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

// Whether the step that reads `slot` may run two-sided (bounds of the header comment; NaN and inf say no).
__device__ bool two_sided(const Geo& g, int slot) {
  const volatile unsigned* s = g.st->slot[slot];
  const volatile unsigned* c = g.st->cst;
  const float r = g.ratio;
  if (!(r >= 0.999999f) || !(dec(c[0]) < 1000.f) || !(dec(c[2]) < 1000.f)) return false;
  const int o = g.self ? 0 : 4;
  const float uf = dec(s[0]), lf = -dec(s[1]), df_max = dec(s[2]), df_min = -dec(s[3]);
  const float ug = dec(s[o]), lg = -dec(s[o + 1]), dg_max = dec(s[o + 2]), dg_min = -dec(s[o + 3]);
  const float wa = dec(c[0]), la = dec(c[1]), wb = dec(c[2]), lb = dec(c[3]);
  const float mass_a = fmaxf(0.f, log2f((float)g.n[0]) + la), mass_b = fmaxf(0.f, log2f((float)g.n[1]) + lb);
  const float row_hi = r * (uf + dg_max) + (r - 1.f) * wb, row_lo = r * (lf + dg_min) - (r - 1.f) * mass_b;
  const float col_hi = r * (ug + df_max) + (r - 1.f) * wa, col_lo = r * (lg + df_min) - (r - 1.f) * mass_a;
  return row_hi + la <= 120.f && row_lo - wa >= -90.f && col_hi + lb <= 120.f && col_lo - wb >= -90.f;
}

// Items of a launch: problem after problem; two-sided: column tile after column tile, all its row tiles (from the
// diagonal on for a self problem); one-sided: side 0 that way, then side 1.
struct Plan {
  int item0[kMaxProblems + 1];
  unsigned two;  // bit per problem
  int ctas;      // CTAs that take part (no more than items)
};
__device__ __forceinline__ int diag_tiles(const Geo& g) { return g.bn / g.bm; }  // row tiles on the diagonal: 1 or 2
// Row tiles of column tile ct of a self problem, and the items before it: column tiles go in pairs (p, last - p), whose
// lengths add up to the same number for every pair, so that short and long runs spread evenly over the CTAs.
__device__ __forceinline__ int self_len(const Geo& g, int ct) { return g.nrt[0] - diag_tiles(g) * ct; }
__device__ __forceinline__ int self_offset(const Geo& g, int ct) {
  const int last = g.nct[0] - 1, pair = self_len(g, 0) + self_len(g, last);
  return 2 * ct <= last ? ct * pair : (last - ct) * pair + self_len(g, last - ct);
}
__device__ __forceinline__ int self_items(const Geo& g) {
  const int last = g.nct[0] - 1, pair = self_len(g, 0) + self_len(g, last);
  return (g.nct[0] / 2) * pair + ((g.nct[0] & 1) ? self_len(g, last / 2) : 0);
}
__device__ int item_count(const Geo& g, bool two) {
  if (g.early && g.ctrl->converged) return 0;
  const int one = g.nct[1] * g.nrt[0];
  if (two) return g.self ? self_items(g) : one;
  return g.self ? one : one + g.nct[0] * g.nrt[1];
}
// By one whole warp.
template <class L>
__device__ void make_plan(const L& P, int slot, int max_ctas, Plan* pl, int lane) {
  int cnt = 0;
  bool two = false;
  if (lane < P.nsub) {
    two = P.two_ok && two_sided(P.sub[lane].geo, slot);
    cnt = item_count(P.sub[lane].geo, two);
  }
  int pre = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, pre, o);
    if (lane >= o) pre += v;
  }
  if (lane < P.nsub) pl->item0[lane + 1] = pre;
  const unsigned mask = __ballot_sync(0xffffffffu, two);
  const int total = __shfl_sync(0xffffffffu, pre, P.nsub - 1);
  if (lane == 0) {
    pl->item0[0] = 0;
    pl->two = mask;
    pl->ctas = total < max_ctas ? total : max_ctas;
  }
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
struct Seg {
  int sub, side, ct, rt, len;
  int strip0;  // first item of the column tile
  bool two;
};
template <class L>
__device__ Seg locate(const L& P, const Plan& pl, int w, int w_end) {
  Seg s;
  s.sub = 0;
  while (pl.item0[s.sub + 1] <= w) ++s.sub;
  const Geo& g = P.sub[s.sub].geo;
  s.two = (pl.two >> s.sub) & 1u;
  s.side = 0;
  int k = w - pl.item0[s.sub], left;
  s.strip0 = pl.item0[s.sub];
  const int r0 = g.nrt[0];
  if (s.two && g.self) {
    const int last = g.nct[0] - 1, pair = self_len(g, 0) + self_len(g, last), p = k / pair;
    k -= p * pair;
    s.ct = p;
    if (k >= self_len(g, p)) {
      k -= self_len(g, p);
      s.ct = last - p;
    }
    s.strip0 += self_offset(g, s.ct);
    s.rt = diag_tiles(g) * s.ct + k;
    left = r0 - s.rt;
  } else {
    int rows = r0;
    if (!s.two && k >= g.nct[1] * r0) {
      k -= g.nct[1] * r0;
      s.strip0 += g.nct[1] * r0;
      s.side = 1;
      rows = g.nrt[1];
    }
    s.ct = k / rows;
    s.rt = k - s.ct * rows;
    s.strip0 += s.ct * rows;
    left = rows - s.rt;
  }
  s.len = left < w_end - w ? left : w_end - w;
  return s;
}

// The run after s, which starts at item w, without the divisions of locate() while the problem and side stay the same.
template <class L>
__device__ __forceinline__ Seg next_run(const L& P, const Plan& pl, Seg s, int w, int w_end) {
  const Geo& g = P.sub[s.sub].geo;
  const bool fold = s.two && g.self;
  const int last = g.nct[1 - s.side] - 1;
  const int ct = !fold ? s.ct + 1 : (2 * s.ct < last ? last - s.ct : last - s.ct + 1);
  if (w >= pl.item0[s.sub + 1] || ct > last || (fold && 2 * s.ct == last)) return locate(P, pl, w, w_end);
  s.strip0 = w;
  s.ct = ct;
  s.rt = fold ? diag_tiles(g) * ct : 0;
  const int left = g.nrt[s.side] - s.rt;
  s.len = left < w_end - w ? left : w_end - w;
  return s;
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

// ------------------------------------------------------------------ the streaming kernel
// KS: the operands do not stay: K chunks of both (32 words; the last one may be partial) share the ring.
template <int NS, bool KS>
__global__ void __launch_bounds__(kThreads, 1) sym_kernel(const __grid_constant__ Launch<NS> P) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  // resident: nfull blocks of 32 words (128-byte swizzle) and ntail of 8 (32-byte swizzle) per operand row
  const uint32_t b_bytes = KS ? 0 : P.nfull * (kBN * 128) + P.ntail * (kBN * 32);
  const uint32_t a_bytes = KS ? kChunk : P.nfull * (128 * 128) + P.ntail * (128 * 32);
  uint8_t* b_smem = base;
  uint8_t* a_smem = b_smem + P.nb * b_bytes;
  float* part = (float*)(a_smem + P.nstage * a_bytes);  // [2 slots][offset | sum][kWG][128]
  uint64_t* bars = (uint64_t*)(part + 2 * 2 * kWG * 128);
  const int A_FULL = 0, A_EMPTY = P.nstage, B_FULL = 2 * P.nstage, B_EMPTY = B_FULL + 2, S_FULL = B_EMPTY + 2,
            S_EMPTY = S_FULL + 2, R_FULL = S_EMPTY + 2, R_EMPTY = R_FULL + 2, DRAIN = R_EMPTY + 2, NBARS = DRAIN + 1;
  uint32_t* tmem_slot = (uint32_t*)(bars + NBARS);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  Plan* plan = (Plan*)(tmem_slot + 2);
  auto bar = [&](int i) { return smem_u32(bars + i); };

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
  pdl_launch();
  pdl_wait();  // everything above overlaps the tail of the previous kernel; its results are read from here on
  if (warp == 2) make_plan(P, P.slot, (int)gridDim.x, plan, lane);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int total = plan->item0[P.nsub], ctas = plan->ctas;
  const bool has_work = (int)blockIdx.x < ctas;
  const int w_begin = has_work ? cta_first(total, ctas, blockIdx.x) : 0;
  const int w_end = has_work ? cta_first(total, ctas, blockIdx.x + 1) : 0;

  if (warp == 0) {
    // ===================== TMA producer =====================
    if (KS && lane == 0 && has_work) {
      int issued = 0;
      bool ok = true;
#pragma unroll 1
      for (int w = w_begin; ok && w < w_end;) {
        const Seg s = locate(P, *plan, w, w_end);
        const Sub& u = P.sub[s.sub];
#pragma unroll 1
        for (int t = 0; ok && t < s.len; ++t)
#pragma unroll 1
          for (int kc = 0; kc < P.nfull; ++kc) {
            const int st = issued % P.nstage;
            if (!(ok = mbar_wait(bar(A_EMPTY + st), ((issued / P.nstage) & 1) ^ 1, abort_flag, 2000))) break;
            mbar_expect_tx(bar(A_FULL + st), kChunk);
            const uint32_t dst = smem_u32(a_smem + st * kChunk);
            tma_load_2d(dst, &u.a_full[s.side], kc * 32, (s.rt + t) * 128, bar(A_FULL + st));
            tma_load_2d(dst + 128 * 128, &u.b_full[s.side], kc * 32, s.ct * kBN, bar(A_FULL + st));
            ++issued;
          }
        w += s.len;
      }
      if (*abort_flag)  // let every copy issued land before the CTA goes away
        for (int j = (issued > P.nstage ? issued - P.nstage : 0); j < issued; ++j)
          mbar_wait_quiet(bar(A_FULL + j % P.nstage), (j / P.nstage) & 1);
    }
    if (!KS && lane == 0 && has_work) {
      int issued = 0, seg = 0, pre = 0;
      bool ok = true;
      auto load_a = [&](const Seg& s, int t) -> bool {
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
      auto load_b = [&](const Seg& s) -> bool {  // column tile of run `seg`
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
      Seg s = locate(P, *plan, w_begin, w_end);
      ok = load_b(s);
#pragma unroll 1
      for (int w = w_begin; ok;) {
#pragma unroll 1
        for (int t = pre; ok && t < s.len; ++t) ok = load_a(s, t);
        w += s.len;
        if (!ok || w >= w_end) break;
        s = next_run(P, *plan, s, w, w_end);
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
    int jt = 0, seg = 0;
    if (KS) {
      int st = 0;
      uint32_t ph = 0;
#pragma unroll 1
      for (; ok && jt < w_end - w_begin; ++jt) {
        const int buf = jt & 1;
        if (!vote(mbar_wait(bar(S_EMPTY + buf), ((jt >> 1) & 1) ^ 1, abort_flag, 2000))) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * kBN);
#pragma unroll 1
        for (int kc = 0; kc < P.nfull; ++kc) {
          if (!vote(mbar_wait(bar(A_FULL + st), ph, abort_flag, 2000))) { ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
            const uint32_t at = smem_u32(a_smem + st * kChunk), al = desc_lo(at), bl = desc_lo(at + 128 * 128);
            const int steps = kc + 1 < P.nfull ? 4 : P.ntail;
#pragma unroll 1
            for (int ks = 0; ks < steps; ++ks)
              umma_step(kc * 4 + ks < P.hs, d_tmem, pack_desc(al + 2 * ks, kDescHi128), pack_desc(bl + 2 * ks, kDescHi128),
                        idesc, idesc_h, (kc | ks) != 0);
            umma_commit(bar(A_EMPTY + st));
            if (kc + 1 == P.nfull) umma_commit(bar(S_FULL + buf));
          }
          __syncwarp();
          if (++st == P.nstage) { st = 0; ph ^= 1; }
        }
      }
    }
#pragma unroll 1
    Seg s;
    if (!KS && has_work) s = locate(P, *plan, w_begin, w_end);
#pragma unroll 1
    for (int w = w_begin; !KS && ok && w < w_end; ++seg) {
      if (w > w_begin) s = next_run(P, *plan, s, w, w_end);
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
      w += s.len;
    }
    __syncwarp();
    if (*abort_flag && lane == 0) {  // wait (bounded) for every MMA issued before TMEM is freed
      umma_commit(bar(DRAIN));
      mbar_wait_quiet(bar(DRAIN), 0);
    }
  } else if (warp == 2) {
    // ===================== row-sum collector: adds the warpgroups' parts, one value per row =====================
    int jt = 0;
    bool ok = true;
    Seg s;
    if (has_work) s = locate(P, *plan, w_begin, w_end);
#pragma unroll 1
    for (int w = w_begin; ok && w < w_end;) {
      if (w > w_begin) s = next_run(P, *plan, s, w, w_end);
      const Geo& g = P.sub[s.sub].geo;
      const size_t at = (size_t)s.ct * g.pad[s.side] + (size_t)s.rt * 128 + lane * 4;
#pragma unroll 1
      for (int i = 0; i < s.len; ++i, ++jt) {
        const int slot = jt & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(bar(R_FULL + slot), (jt >> 1) & 1, abort_flag, 1000))) {
          ok = false;
          break;
        }
        const float4* ps = reinterpret_cast<const float4*>(part + (slot * 2 + 1) * kWG * 128) + lane;
        float4 v[kWG];
#pragma unroll
        for (int k = 0; k < kWG; ++k) v[k] = ps[k * 32];
        if (s.two) {
          float4 o;
          o.x = (v[0].x + v[1].x) + (v[2].x + v[3].x);
          o.y = (v[0].y + v[1].y) + (v[2].y + v[3].y);
          o.z = (v[0].z + v[1].z) + (v[2].z + v[3].z);
          o.w = (v[0].w + v[1].w) + (v[2].w + v[3].w);
          *reinterpret_cast<float4*>(g.rp_s[0] + at + (size_t)i * 128) = o;
        } else {
          const float4* pm = reinterpret_cast<const float4*>(part + slot * 2 * kWG * 128) + lane;
          float4 m[kWG];
#pragma unroll
          for (int k = 0; k < kWG; ++k) m[k] = pm[k * 32];
          auto join = [&](float m0, float m1, float m2, float m3, float s0, float s1, float s2, float s3, float& sum) {
            const float top = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
            sum = (s0 * ex2(m0 - top) + s1 * ex2(m1 - top)) + (s2 * ex2(m2 - top) + s3 * ex2(m3 - top));
            return top;
          };
          float4 om, os;
          om.x = join(m[0].x, m[1].x, m[2].x, m[3].x, v[0].x, v[1].x, v[2].x, v[3].x, os.x);
          om.y = join(m[0].y, m[1].y, m[2].y, m[3].y, v[0].y, v[1].y, v[2].y, v[3].y, os.y);
          om.z = join(m[0].z, m[1].z, m[2].z, m[3].z, v[0].z, v[1].z, v[2].z, v[3].z, os.z);
          om.w = join(m[0].w, m[1].w, m[2].w, m[3].w, v[0].w, v[1].w, v[2].w, v[3].w, os.w);
          *reinterpret_cast<float4*>(g.rp_m[s.side] + at + (size_t)i * 128) = om;
          *reinterpret_cast<float4*>(g.rp_s[s.side] + at + (size_t)i * 128) = os;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(R_EMPTY + slot));
      }
      w += s.len;
    }
  } else if (warp >= 4) {
    // ===================== soft-max warpgroups =====================
    const int wg = (warp - 4) >> 2, q = warp & 3;  // columns [64 wg, 64 wg + 64) of a tile; TMEM lane quarter
    const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + wg * 64;
    const int trow = q * 32 + lane;
    bool ok = true;
    int jt = 0;
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
    Seg s;
    if (has_work) s = locate(P, *plan, w_begin, w_end);
#pragma unroll 1
    for (int w = w_begin; w < w_end;) {
      if (w > w_begin) s = next_run(P, *plan, s, w, w_end);
      const Geo& g = P.sub[s.sub].geo;
      const float pair = P.sub[s.sub].scale2 / pair_scale(g.scales.range);  // exact: a power of two
      if (s.two) {
        const float scale = pair;
        const u64 sc = pk(scale, scale);
        // row tiles that lie on the diagonal of a self problem: row sums only (both halves of each pair are there)
        int diag = g.self ? 2 * s.ct + 2 - s.rt : 0;
        u64 acc[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = 0ull;
        uint32_t ra[8], rb[8];
        // the first scores of a tile load while the last ones of the tile before are worked on
        if (ok && (ok = wait_tile(jt))) tmem_ld8_nowait(lane_addr + (uint32_t)((jt & 1) * kBN), ra);
#pragma unroll 1
        for (int i = 0; ok && i < s.len; ++i, ++jt) {
          const uint32_t src = lane_addr + (uint32_t)((jt & 1) * kBN);
          u64 rs0 = 0ull, rs1 = 0ull;
          auto eat = [&](const uint32_t (&r)[8], int c) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              float z0, z1;
              upk(mul2(pk(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1])), sc), z0, z1);
              const u64 e = pk(ex2(z0), ex2(z1));
              acc[c * 4 + k] = add2(acc[c * 4 + k], e);
              if (k & 1) rs1 = add2(rs1, e); else rs0 = add2(rs0, e);
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
          release_tile();
          bool more = i + 1 < s.len;
          if (more && !wait_tile(jt + 1)) more = ok = false;
          if (more) tmem_ld8_nowait(lane_addr + (uint32_t)(((jt + 1) & 1) * kBN), ra);
          eat(rb, 7);
          float a0, a1, a2, a3;
          upk(rs0, a0, a1);
          upk(rs1, a2, a3);
          if (!post(0.f, (a0 + a1) + (a2 + a3))) ok = false;
          if (!ok) break;
          if (diag > 0) {
            --diag;
#pragma unroll
            for (int k = 0; k < 32; ++k) acc[k] = 0ull;
          }
        }
        // End of the run: one sum per column and warp.
        float v[64];
#pragma unroll
        for (int k = 0; k < 32; ++k) upk(acc[k], v[2 * k], v[2 * k + 1]);
        warp_columns(v, lane);
        if (ok) {  // one row of partials per warp (32 rows of each tile): no barrier at the end of a run
          const int piece = s.strip0 >= w_begin ? 0 : (int)blockIdx.x - cta_of(total, ctas, s.strip0);
          float* to = g.cp + (size_t)(piece * 4 + q) * g.pad[1] + s.ct * kBN + wg * 64 + 2 * lane;
          *reinterpret_cast<float2*>(to) = make_float2(v[0], v[1]);
        }
      } else {
        const bool wide = wide_range(g.scales);
#pragma unroll 1
        for (int i = 0; ok && i < s.len; ++i, ++jt) {
          if (!(ok = wait_tile(jt))) break;
          const uint32_t src = lane_addr + (uint32_t)((jt & 1) * kBN);
          const float scale = wide ? P.sub[s.sub].scale2 * g.scales.inv[s.side][(s.rt + i) * 128 + trow] : pair;
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
      w += s.len;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
  if (tid == 0 && *abort_flag) atomicExch(&g_sym_error, 1);
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
  uint32_t* tmem_slot = (uint32_t*)(bars + NBARS);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  Plan* plan = (Plan*)(tmem_slot + 2);
  auto bar = [&](int i) { return smem_u32(bars + i); };
  const Sub& u = P.sub[0];
  const Geo& g = u.geo;

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
  pdl_launch();
  pdl_wait();
  if (warp == 2) make_plan(P, P.slot, (int)gridDim.x, plan, lane);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int total = plan->item0[1];
  const bool two = plan->two & 1u;
  // Item k: (side, row tile, column tile).
  auto locate_tile = [&](int k, int& side, int& rt, int& ct) {
    side = 0;
    if (two && g.self) {
      const Seg s = locate(P, *plan, k, k + 1);
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
      int issued = 0;
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
    int s = 0, jt = 0;
    uint32_t ph = 0;
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
    const float pair = u.scale2 / pair_scale(g.scales.range);  // exact: a power of two
    const bool wide = wide_range(g.scales);
    bool ok = true;
    int jt = 0;
#pragma unroll 1
    for (int k = blockIdx.x; k < total; k += gridDim.x, ++jt) {  // also after an abort: every warp takes every barrier
      int side, rt, ct;
      locate_tile(k, side, rt, ct);
      const int buf = h * NBUF + jt % NBUF, sl = jt & 1;
      if (ok) ok = mbar_wait(bar(S_FULL + buf), (jt / NBUF) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok) != 0;
      const float scale = wide ? u.scale2 * g.scales.inv[side][rt * BM + trow] : pair;
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

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  if (tid == 0 && *abort_flag) atomicExch(&g_sym_error, 1);
}

// ------------------------------------------------------------------ staging and finalising
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
  return fabs(pot / eps + own) * 1.4426950408889634 <= 1048576.0;
}

// Adds the partial sums of a step, updates the potentials in place (rounded once from fp64), stages the biases of
// the next step and records the ranges that decide how it runs. One block per 32 points, eight warps share the
// partials of each. Bound by latency: a few loads per thread behind the streaming kernel.
template <int NS>
__global__ void __launch_bounds__(256) sym_finalize_kernel(const __grid_constant__ FinLaunch<NS> P) {
  __shared__ Plan plan;
  __shared__ float red_m[8][32], red_s[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch();
  pdl_wait();
  const FinSub& u = P.sub[blockIdx.y];
  const Geo& g = u.geo;
  unsigned* next = g.st->slot[(P.slot + 1) % 3];
  if (g.early && g.ctrl->converged) {  // the range record must not outlive the potentials it describes
    if (blockIdx.x == 0 && threadIdx.x == 0) next[0] = enc(INFINITY);
    return;
  }
  const int nb0 = (g.n[0] + 31) / 32, nb1 = g.self ? 0 : (g.n[1] + 31) / 32;
  if ((int)blockIdx.x >= nb0 + nb1) return;
  const int c = (int)blockIdx.x < nb0 ? 0 : 1;
  const int i0 = ((int)blockIdx.x - (c ? nb0 : 0)) * 32, i = i0 + lane;
  // what the last warp standing needs is fetched together with the words of the plan
  float pot_i = 0.f, logw_i = 0.f, sq_i = 0.f, unit_i = 1.f;
  if (warp == 0) {
    if (i < g.n[c]) {
      unit_i = bias_factor(g.scales, wide_range(g.scales), c, i);
      pot_i = __ldcg(u.pot[c] + i);
      logw_i = __ldg(u.logw[c] + i);
      if (u.shiftcoef[c] != 0.f) sq_i = __ldcg(u.sq[c] + i);
    }
    make_plan(P, P.slot, P.ctas, &plan, lane);
  }
  __syncthreads();
  const bool two = (plan.two >> blockIdx.y) & 1u;
  const int pad = g.pad[c];

  if (two) {
    int k_rows = 0, k_cols = 0;  // partials from row sums / from column sums
    const int ct = i0 / g.bn;
    size_t col0 = 0;
    if (c == 0) k_rows = g.self ? ct + 1 : g.nct[1];
    if (c == 1 || g.self) {
      if (g.by_tile) {
        col0 = g.self ? diag_tiles(g) * (ct + 1) : 0;
        k_cols = g.nrt[0] - (int)col0;
      } else {
        const int total = plan.item0[P.nsub];
        const int len = g.self ? self_len(g, ct) : g.nrt[0];
        const int first = plan.item0[blockIdx.y] + (g.self ? self_offset(g, ct) : ct * g.nrt[0]);
        k_cols = 4 * (cta_of(total, plan.ctas, first + len - 1) - cta_of(total, plan.ctas, first) + 1);
      }
    }
    const int pad1 = g.pad[1];
    // eight independent loads in flight per thread: at 50,000 points a side there are 200 partials per row, and the
    // kernel is bound by their latency (100 us of a 1.56 ms step with two at a time)
    auto gather = [&](const float* from, int count, size_t pitch) {
      float t[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int k = warp; k < count; k += 64) {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (k + 8 * e < count) t[e] += __ldcg(from + (size_t)(k + 8 * e) * pitch);
      }
      return ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
    };
    red_m[warp][lane] = 0.f;
    red_s[warp][lane] = gather(g.rp_s[0] + i, k_rows, g.pad[0]) + gather(g.cp + col0 * pad1 + i, k_cols, pad1);
  } else {
    const int parts = g.nct[g.self ? 0 : 1 - c];
    float m = -INFINITY, s = 0.f;
    const float *pm = g.rp_m[c] + i, *ps = g.rp_s[c] + i;
#pragma unroll 8
    for (int k = warp; k < parts; k += 8) m = fmaxf(m, __ldcg(pm + (size_t)k * pad));
#pragma unroll 4
    for (int k = warp; k < parts; k += 8) s += __ldcg(ps + (size_t)k * pad) * ex2(__ldcg(pm + (size_t)k * pad) - m);
    red_m[warp][lane] = m;
    red_s[warp][lane] = s;
  }
  __syncthreads();
  if (warp != 0) return;
  float m = red_m[0][lane], s;
#pragma unroll
  for (int k = 1; k < 8; ++k) m = fmaxf(m, red_m[k][lane]);
  if (two) {
    s = ((red_s[0][lane] + red_s[1][lane]) + (red_s[2][lane] + red_s[3][lane])) +
        ((red_s[4][lane] + red_s[5][lane]) + (red_s[6][lane] + red_s[7][lane]));
  } else {
    s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (red_s[k][lane] != 0.f) s += red_s[k][lane] * ex2(red_m[k][lane] - m);
  }
  float st_u = -INFINITY, st_l = -INFINITY, st_dx = -INFINITY, st_dn = -INFINITY;
  if (i < g.n[c]) {
    // log2 of the weighted sum with the point's own bias inside; the candidate takes that bias out again
    const float l2 = m + log2f(fmaxf(s, 1e-40f));
    const double old = (double)pot_i, lw = (double)logw_i, own = own_logw(lw);
    const bool inside = own_inside(old, own, u.eps);
    const double cand =
        (double)u.damp[c] * ((inside ? old : 0.0) + u.eps * ((inside ? own : 0.0) - (double)l2 * 0.69314718055994530942));
    double v = (1.0 - (double)u.w) * old + (double)u.w * cand;
    if (u.shiftcoef[c] != 0.f) v -= (double)u.shiftcoef[c] * (double)sq_i;
    const float now = (float)v;
    u.pot[c][i] = now;
    const size_t at = (size_t)i * P.kp + P.kc;
    const double to_unit = u.inv2cs * (double)unit_i;
    const bool inside_next = own_inside((double)now, own, u.eps_next);
    write_bias(u.opA[c] + at + 3, inside_next ? ((double)now + own * u.eps_next) * to_unit : 0.0);
    write_bias(u.opB[c] + at, ((double)now + lw * u.eps_next) * to_unit);
    const float big_l = (float)((double)l2 - own * 1.4426950408889634);
    const float dlt = (float)(((double)now - old) * u.log2e_eps);
    st_u = big_l + dlt;
    st_l = -st_u;
    st_dx = dlt;
    st_dn = -dlt;
    // no bound: the next step runs one-sided
    if (!(fabsf(st_u) < 1e30f) || !(fabsf(dlt) < 1e30f) || !inside || !inside_next) st_u = INFINITY;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    st_u = fmaxf(st_u, __shfl_xor_sync(0xffffffffu, st_u, o));
    st_l = fmaxf(st_l, __shfl_xor_sync(0xffffffffu, st_l, o));
    st_dx = fmaxf(st_dx, __shfl_xor_sync(0xffffffffu, st_dx, o));
    st_dn = fmaxf(st_dn, __shfl_xor_sync(0xffffffffu, st_dn, o));
  }
  if (lane < 4) {
    const float v = lane == 0 ? st_u : (lane == 1 ? st_l : (lane == 2 ? st_dx : st_dn));
    atomicMax(next + 4 * c + lane, enc(v));
  }
  if (blockIdx.x == 0) {
    if (lane == 31) g.ctrl->iters_used += 1;
    if (lane == 30 && two) atomicAdd(&g_sym_two_sided, 1ull);
    if (lane >= 8 && lane < 16) g.st->slot[(P.slot + 2) % 3][lane - 8] = 0u;
  }
}

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

template <int NS>
__global__ void sym_reset_kernel(const __grid_constant__ StageLaunch<NS> P) {
  const int i = threadIdx.x;
  if (i >= P.nsub) return;
  State* st = P.sub[i].st;
  for (int k = 0; k < 8; ++k) {
    st->slot[0][k] = enc(INFINITY);  // nothing is known about the first step: it runs one-sided
    st->slot[1][k] = st->slot[2][k] = 0u;
  }
  for (int k = 0; k < 4; ++k) st->cst[k] = 0u;
  for (int k = 0; k < kRangeWords; ++k) st->range[k] = 0u;
  Ctrl* c = P.sub[i].ctrl;
  c->delta_bits = 0u; c->converged = 0; c->have_prev = 0; c->iters_used = 0;
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

// Stages the biases again for a step at eps (FinSub::eps_next), from the potentials as they are. One thread per point.
__global__ void sym_rebias_kernel(const __grid_constant__ FinLaunch<1> P) {
  const FinSub& u = P.sub[0];
  const Geo& g = u.geo;
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
  pdl_wait();
  const EmitJobs::Job& j = P.job[blockIdx.y];
  const int c = blockIdx.z, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < j.n[c] && j.out[c]) j.out[c][i] = j.pot[c][i] + j.sq[c][i];
}

// ------------------------------------------------------------------ host side
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

struct Carve {
  char* base;
  size_t off = 0;
  template <typename T>
  T* take(size_t count) {
    const size_t o = off;
    off += (count * sizeof(T) + 1023) & ~size_t(1023);
    return base ? reinterpret_cast<T*>(base + o) : nullptr;
  }
};

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

template <typename K, typename A>
cudaError_t launch_pdl(K kern, dim3 grid, int threads, size_t smem, cudaStream_t st, const A& arg) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, arg);
}

template <int NS>
cudaError_t step_n(const Step* s, int cnt, int t, cudaStream_t st) {
  const Problem& p0 = *s[0].p;
  const Shape sh = plan_shape(p0.n[0], p0.n[1], p0.d, p0.prec, 3 * p0.lab.V);
  Launch<NS> lp;
  FinLaunch<NS> fp;
  lp.nsub = fp.nsub = cnt;
  lp.nfull = sh.nfull; lp.ntail = sh.ntail; lp.nstage = sh.nstage;
  lp.hs = sh.hs;
  lp.nb = sh.nb;
  lp.slot = fp.slot = t % 3;
  fp.kc = sh.kc; fp.kp = sh.kp;
  long long most = 0;
  int blocks = 1;
  for (int i = 0; i < cnt; ++i) {
    const Problem& p = *s[i].p;
    Geo g = p.geo;
    g.early = s[i].early ? 1 : 0;
    g.ratio = (float)(s[i].eps_prev / s[i].eps);
    Sub& u = lp.sub[i];
    for (int k = 0; k < 2; ++k) {
      u.a_full[k] = p.map[4 * k]; u.a_tail[k] = p.map[4 * k + 1];
      u.b_full[k] = p.map[4 * k + 2]; u.b_tail[k] = p.map[4 * k + 3];
    }
    u.geo = g;
    u.scale2 = (2.0f * p.cs_dot) * (1.0f / (float)s[i].eps) * kLog2e;
    FinSub& f = fp.sub[i];
    f.geo = g;
    for (int k = 0; k < 2; ++k) {
      f.pot[k] = p.pot[k]; f.logw[k] = p.logw[k]; f.sq[k] = p.sq[k]; f.opA[k] = p.opA[k]; f.opB[k] = p.opB[k];
      f.damp[k] = s[i].damp[k];
      f.shiftcoef[k] = s[i].damp[k] < 1.f ? s[i].w * (1.f - s[i].damp[k]) : 0.f;
    }
    f.eps = (float)s[i].eps;
    f.eps_next = (float)s[i].eps_next;
    f.inv2cs = 0.5 / (double)p.cs_dot;
    f.log2e_eps = 1.4426950408889634 / f.eps;
    f.w = s[i].w;
    most += (long long)g.nct[1] * g.nrt[0] + (p.self ? 0 : (long long)g.nct[0] * g.nrt[1]);
    const int nb = tiles(p.n[0], 32) + (p.self ? 0 : tiles(p.n[1], 32));
    blocks = nb > blocks ? nb : blocks;
  }
  int ctas = tc::detail::free_ctas();
  if (ctas > kMaxCtas) ctas = kMaxCtas;
  // With a CTA for every one-sided item there is nothing to share: both sides run next to each other on SMs that
  // would idle, without the column reduction and without a bound on the range.
  lp.two_ok = fp.two_ok = most > ctas;
  if (most < ctas) ctas = (int)most;
  fp.ctas = ctas;
  auto go = [&](auto kern, int threads, const auto& arg) {
    cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    return r == cudaSuccess ? launch_pdl(kern, dim3(ctas), threads, sh.smem, st, arg) : r;
  };
  cudaError_t e = cudaErrorInvalidValue;
  if (sh.kind == RESIDENT) e = go(sym_kernel<NS, false>, kThreads, lp);
  if (sh.kind == STREAMED) e = go(sym_kernel<NS, true>, kThreads, lp);
  if constexpr (NS == 1) {
    if (sh.kind == WIDE) e = go(sym_wide_kernel<2, 256, 1, 2>, 128 + 512, lp);
    if (sh.kind == SMALL) e = go(sym_wide_kernel<1, 128, 2, 4>, 128 + 512, lp);
  }
  if (e == cudaSuccess) e = launch_pdl(sym_finalize_kernel<NS>, dim3(blocks, cnt), 256, 0, st, fp);
  count_launches(2);
  return e;
}

template <int NS>
cudaError_t stage_n(Problem* const* p, const double* eps0, int cnt, cudaStream_t st) {
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
    u.cs_sq = q.cs_sq; u.eps = (float)eps0[i]; u.inv2cs = 0.5 / (double)q.cs_dot;
    u.self = q.self ? 1 : 0; u.st = q.geo.st; u.ctrl = q.ctrl;
    blocks[0] = q.geo.pad[0] / 8 > blocks[0] ? q.geo.pad[0] / 8 : blocks[0];
    if (!q.self) blocks[1] = q.geo.pad[1] / 8 > blocks[1] ? q.geo.pad[1] / 8 : blocks[1];
  }
  sym_reset_kernel<NS><<<1, 32, 0, st>>>(lp);
  count_launches(1);
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

cudaError_t stage(Problem* const* p, const double* eps0, int cnt, cudaStream_t st) {
  if (cnt < 1 || cnt > kMaxProblems) return cudaErrorInvalidValue;
  if (cnt == 1) return stage_n<1>(p, eps0, cnt, st);
  if (cnt <= 3) return stage_n<3>(p, eps0, cnt, st);
  return stage_n<kMaxProblems>(p, eps0, cnt, st);
}

cudaError_t step(const Step* s, int cnt, int t, cudaStream_t st) {
  if (cnt < 1 || cnt > kMaxProblems) return cudaErrorInvalidValue;
  bool alone = false;  // one launch per problem: long contractions, and tile shapes that differ between problems
  for (int i = 0; i < cnt; ++i) alone = alone || s[i].p->kind >= WIDE || s[i].p->kind != s[0].p->kind;
  if (alone && cnt > 1) {
    for (int i = 0; i < cnt; ++i) {
      cudaError_t e = step_n<1>(s + i, 1, t, st);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  if (cnt == 1) return step_n<1>(s, cnt, t, st);
  if (cnt <= 3) return step_n<3>(s, cnt, t, st);
  return step_n<kMaxProblems>(s, cnt, t, st);
}

cudaError_t rebias(const Problem& p, double eps, cudaStream_t st) {
  FinLaunch<1> fp;
  fp.kc = p.kc; fp.kp = p.kp;
  FinSub& f = fp.sub[0];
  f.geo = p.geo;
  for (int k = 0; k < 2; ++k) {
    f.pot[k] = p.pot[k]; f.logw[k] = p.logw[k]; f.opA[k] = p.opA[k]; f.opB[k] = p.opB[k];
  }
  f.eps_next = (float)eps;
  f.inv2cs = 0.5 / (double)p.cs_dot;
  const int rows = p.n[0] > p.n[1] ? p.n[0] : p.n[1];
  sym_rebias_kernel<<<dim3((rows + 255) / 256, p.self ? 1 : 2), 256, 0, st>>>(fp);
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
  return launch_pdl(sym_emit_kernel, dim3((rows + 255) / 256, cnt, 2), 256, 0, st, jobs);
}

int kernel_of(int n, int m, int d, int prec, int nlab) {
  const int kind = plan_shape(n, m, d, prec, nlab).kind;
  return kind == RESIDENT ? 1 : (kind == STREAMED ? 2 : (kind == WIDE ? 3 : 4));
}

long long two_sided_steps() {
  unsigned long long v = 0;
  return cudaMemcpyFromSymbol(&v, g_sym_two_sided, sizeof(v)) == cudaSuccess ? (long long)v : -1;
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
