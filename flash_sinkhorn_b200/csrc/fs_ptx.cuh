// Inline-PTX wrappers for the sm_100a tensor-core engines (tcgen05 / TMEM / TMA / mbarrier) and the few
// constants the kernels share. Included by the translation units that hold such kernels; everything is
// internal to the including file.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "fs_common.cuh"

namespace fs {
namespace tc {
namespace {

constexpr float kMaskBias = -1.2676506e30f;  // -2^100: bias of padded columns (finite: survives the MMA)
constexpr float kRunInit = -1.0e30f;         // initial running max (above the mask, below any real logit)
constexpr long long kSpinLimit = 1ll << 28;  // ~0.14 s of SM cycles per wait (a tile takes microseconds)
constexpr int kSmemMin = 120 * 1024;         // force one CTA per SM (TMEM is allocated per CTA)
constexpr int kSmemMax = 227 * 1024;

// Initial running maximum of scores that `scale` > 0 turns into exponents: their product stays finite, so that a stretch of
// padded columns (whose scores may reach -inf as exponents) adds nothing at an offset that compares and subtracts.
__device__ __forceinline__ float run_init(float scale) { return fmaxf(kRunInit, -1.0e38f / scale); }

// ------------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// try_wait with a suspend-time hint: the hardware parks the thread until the phase completes or about
// `ns` nanoseconds pass, so a waiting single-lane role neither burns issue slots nor wakes up late.
__device__ __forceinline__ bool mbar_try_wait_hint(uint32_t bar, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(ns)
      : "memory");
  return ok != 0;
}
// Bounded wait. Returns false (and raises *abort_flag) if the budget runs out or another
// thread of the CTA already aborted. `park_ns` > 0 selects the parking form of try_wait (producer / MMA
// lanes, which spend most of their time waiting and share a scheduler with soft-max warps).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          unsigned park_ns = 0) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
    if (park_ns ? mbar_try_wait_hint(bar, parity, park_ns) : mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > kSpinLimit) {
      *abort_flag = 1;
      return false;
    }
  }
}
// Teardown wait: bounded, ignores the abort flag (used to let in-flight copies / MMAs land).
__device__ __forceinline__ void mbar_wait_quiet(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > kSpinLimit) return;
  }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// One lane of a converged warp (elect.sync). The MMA-issuing warps run their loops with all 32 lanes, so that
// descriptor and address arithmetic is warp-uniform (the compiler can keep it in uniform registers, which is
// where tcgen05 instructions take their operands), and only the instruction itself is issued by one lane.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// Registers of a CTA of 128 + 512 threads, launched with 96 each: 32 for the service warps 0..3, 112 for the soft-max warps
// (128 x 32 + 512 x 112 = 640 x 96). Executed by whole warpgroups.
__device__ __forceinline__ void registers_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 32;"); }
__device__ __forceinline__ void registers_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 112;"); }

// D[tmem] (+)= A[smem desc] x B[smem desc]^T, M=128, N from idesc, K=8 (tf32)
__device__ __forceinline__ void umma_tf32(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  // the wait takes r[] as read-write operands: no use of the data can be scheduled above it
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                 "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                 "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Same load without the wait: the caller overlaps it with arithmetic and calls tmem_ld_wait() before use.
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// Wait for the outstanding TMEM loads. The destination registers are passed through the asm as
// read-write operands so that no use of them can be scheduled above the wait.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                 "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                 "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// Packed pairs of floats (one issue slot for two lanes of arithmetic).
typedef unsigned long long u64;
__device__ __forceinline__ u64 pk(float lo, float hi) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void upk(u64 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
  u64 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
  u64 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// Shared-memory matrix descriptor, K-major operand (PTX "tcgen05 matrix descriptor"):
//   [0,14) start address >> 4, [16,30) leading byte offset >> 4 (unused for swizzled K-major: 1),
//   [32,46) stride byte offset >> 4 (distance between 8-row groups), [46,48) version = 1,
//   [61,64) layout: 2 = 128-byte swizzle, 6 = 32-byte swizzle.
// It is assembled from a running low word (address >> 4, leading-offset field = 1) and a constant high
// word, which lets the MMA-issuing lane advance operands with one integer add.
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (1u << 16); }
__device__ __forceinline__ uint64_t pack_desc(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}
constexpr uint32_t kDescHi128 = (1024u >> 4) | (1u << 14) | (2u << 29);  // 8-row groups 1024 B apart, 128 B swizzle
constexpr uint32_t kDescHi32 = (256u >> 4) | (1u << 14) | (6u << 29);    // 8-row groups 256 B apart, 32 B swizzle

// Instruction descriptor for kind::tf32, fp32 accumulate, both operands K-major, M=128:
//   [4,6) D format = 1 (f32), [7,10) A format = 2 (tf32), [10,13) B format = 2 (tf32),
//   [17,23) N >> 3, [24,29) M >> 4.
__host__ __device__ constexpr uint32_t make_idesc(int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void umma_tf32_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// kind::f16 with fp16 operands and an fp32 accumulator: K = 16 per instruction over the same 32 bytes of an operand
// row that hold 8 TF32 values, at the same clocks - twice the products per instruction and per byte.
__host__ __device__ constexpr uint32_t make_idesc_f16(int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// One 32-byte K step of an operand row: 16 scaled fp16 coordinates (half) or 8 TF32 columns.
__device__ __forceinline__ void umma_step(bool half, uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc_tf32,
                                          uint32_t idesc_f16, uint32_t accumulate) {
  if (half) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc_f16), "r"(accumulate)
        : "memory");
  } else {
    umma_tf32(d_tmem, adesc, bdesc, idesc_tf32, accumulate);
  }
}

// Scaled fp16 coordinates. Float bits of a magnitude -> k of the power of two that brings it to [2^14, 2^15): there an
// fp16 carries the 11 significant bits of a TF32 value, and a pair of them 22, over some octaves below.
__device__ __forceinline__ int scale_exponent(unsigned bits, int lo, int hi) {
  const int e = (int)(bits >> 23);
  if (bits == 0u || e >= 255) return 0;
  const int k = 14 - (e - 127);
  return k > hi ? hi : (k < lo ? lo : k);
}
__device__ __forceinline__ float power_of_two(int k) { return __uint_as_float((unsigned)(k + 127) << 23); }
// ONE scale per cloud, from its largest |coordinate|: the product of two clouds' scales divides the logit scale. The
// limits keep that product well inside the exponent range of the bias columns it multiplies.
__device__ __forceinline__ float cloud_scale(unsigned amax_bits) { return power_of_two(scale_exponent(amax_bits, -50, 30)); }
__device__ __forceinline__ float pair_scale(const unsigned* range) {
  return range ? cloud_scale(range[0]) * cloud_scale(range[1]) : 1.f;
}
// A scale of its own for a point. The upper limit leaves bias columns of up to 2^30 against two tiny points.
__device__ __forceinline__ int point_exponent(unsigned max_bits) { return scale_exponent(max_bits, -113, 48); }

// Whether one scale per cloud is enough: it has to carry the largest coordinate without overflow and the largest
// coordinate of EVERY point (other than zeros) within `octaves` below it, the range over which the point keeps the
// significant bits of TF32 pieces. A point far from the rest, an infinity or a NaN would take them from all others.
__device__ __forceinline__ bool narrow_cloud(unsigned top, unsigned low_complement, int octaves) {
  const int k = scale_exponent(top, -50, 30) - 127;
  return top == 0u || (top < 0x7f800000u && (int)(top >> 23) + k <= 14 && (int)(~low_complement >> 23) + k >= 14 - octaves);
}
// Where it is not enough for either cloud, every point has its own scale in both roles, ones, bias and label columns carry
// it along, and each score is divided by the two points' scales where it leaves the accumulator.
__device__ __forceinline__ bool wide_range(const OperandScales& s) { return s.range && s.range[4] != 0u; }
// What the coordinates of point r of a cloud are multiplied by; its column of ones; its bias and label columns.
__device__ __forceinline__ float coord_factor(const OperandScales& s, bool wide, int cloud, int r) {
  return !s.range ? 1.f : (wide ? 1.f / s.inv[cloud][r] : cloud_scale(s.range[cloud]));
}
__device__ __forceinline__ float ones_factor(const OperandScales& s, bool wide, int cloud, int r) {
  return wide ? 1.f / s.inv[cloud][r] : 1.f;
}
__device__ __forceinline__ float bias_factor(const OperandScales& s, bool wide, int cloud, int r) {
  return wide ? 1.f / s.inv[cloud][r] : pair_scale(s.range);
}
// 32 scores against consecutive columns whose 1 / scale are at inv (the same addresses for the whole warp).
__device__ __forceinline__ void unscale_columns(uint32_t (&r)[32], const float* inv) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(inv) + i);
    r[4 * i] = __float_as_uint(__uint_as_float(r[4 * i]) * f.x);
    r[4 * i + 1] = __float_as_uint(__uint_as_float(r[4 * i + 1]) * f.y);
    r[4 * i + 2] = __float_as_uint(__uint_as_float(r[4 * i + 2]) * f.z);
    r[4 * i + 3] = __float_as_uint(__uint_as_float(r[4 * i + 3]) * f.w);
  }
}
// Coordinate column k (32-bit word) of a staged operand row, row role (va) and column role (vb). parts = 1: the
// coordinates to 11 significant bits; parts = 3: [hi | hi | lo] against [hi | lo | hi], 22 bits and a product that
// drops only lo.lo. hs > 0: hs K steps of 16 scaled fp16 values, two per word, every part padded to whole steps;
// hs == 0: TF32 values, one per word.
__device__ __forceinline__ void stage_coord(const float* row, int k, int d, int parts, int hs, float scale, float& va,
                                            float& vb) {
  if (hs > 0) {
    const int words = hs * 8 / parts, part = k / words, c = 2 * (k - part * words);
    // rounded as TF32 values first (ties away from zero): the conversions of the scaled pieces are then exact
    const float x0 = c < d ? row[c] : 0.f, x1 = c + 1 < d ? row[c + 1] : 0.f, h0 = to_tf32(x0), h1 = to_tf32(x1);
    const __half2 hi = __floats2half2_rn(h0 * scale, h1 * scale);
    const __half2 lo = __floats2half2_rn(to_tf32(x0 - h0) * scale, to_tf32(x1 - h1) * scale);
    const __half2 a = part == 2 ? lo : hi, b = part == 1 ? lo : hi;
    va = __uint_as_float(*reinterpret_cast<const unsigned*>(&a));
    vb = __uint_as_float(*reinterpret_cast<const unsigned*>(&b));
  } else {
    const int part = k / d;
    const float x = row[k - part * d], hi = to_tf32(x), lo = to_tf32(x - hi);
    va = part == 2 ? lo : hi;
    vb = part == 1 ? lo : hi;
  }
}
// Largest |coordinate| of every row of x [rows, d]: 1 / point scale to inv [pad] (1 for padded rows; null: not wanted) and,
// unless range is null, the range over all rows into its words `cloud` and 2 + cloud, as float bits (NaN and inf come out
// above every finite value). range starts at zero; the last of `looking` blocks, over both clouds, decides whether it is
// wide. By whole blocks, `block` of `blocks`. Bound by the read of the cloud: 256 KB and more in flight per SM.
__device__ __forceinline__ void row_ranges(const float* x, int rows, int pad, int d, int block, int blocks, float* inv,
                                           unsigned* range, int cloud, int looking, int octaves) {
  const int lane = threadIdx.x & 31, warps = (int)blockDim.x >> 5, warp = (int)threadIdx.x >> 5;
  unsigned hi = 0u, lo = 0u;
  auto bits = [&](long long r, int k) { return __float_as_uint(__ldg(x + (size_t)r * d + k)) & 0x7fffffffu; };
  auto put = [&](unsigned m) {
    hi = m > hi ? m : hi;
    lo = m && ~m > lo ? ~m : lo;
  };
  if (d <= 64) {  // eight short rows at a time
    for (long long r0 = (long long)(block * warps + warp) * 8; r0 < pad; r0 += (long long)blocks * warps * 8) {
      unsigned m[8], mine = 0u;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const bool in = r0 + u < rows;
        const unsigned a = in && lane < d ? bits(r0 + u, lane) : 0u, b = in && lane + 32 < d ? bits(r0 + u, lane + 32) : 0u;
        m[u] = a > b ? a : b;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        m[u] = __reduce_max_sync(0xffffffffu, m[u]);
        put(m[u]);
        mine = lane == u ? m[u] : mine;
      }
      if (inv && lane < 8 && r0 + lane < pad) inv[r0 + lane] = power_of_two(-point_exponent(mine));
    }
  } else {
    for (long long r = block * warps + warp; r < pad; r += (long long)blocks * warps) {
      unsigned m = 0u;
      if (r < rows) {
#pragma unroll 8
        for (int k = lane; k < d; k += 32) {
          const unsigned b = bits(r, k);
          m = b > m ? b : m;
        }
      }
      m = __reduce_max_sync(0xffffffffu, m);
      put(m);
      if (inv && lane == 0) inv[r] = power_of_two(-point_exponent(m));
    }
  }
  if (!range) return;
  __shared__ unsigned red[2][32];
  if (lane == 0) {
    red[0][warp] = hi;
    red[1][warp] = lo;
  }
  __syncthreads();
  if (warp == 0) {
    hi = __reduce_max_sync(0xffffffffu, lane < warps ? red[0][lane] : 0u);
    lo = __reduce_max_sync(0xffffffffu, lane < warps ? red[1][lane] : 0u);
    if (lane == 0) {
      if (hi) atomicMax(range + cloud, hi);
      if (lo) atomicMax(range + 2 + cloud, lo);
      __threadfence();
      if (atomicAdd(range + 5, 1u) == (unsigned)looking - 1u) {
        const volatile unsigned* w = range;
        range[4] = narrow_cloud(w[0], w[2], octaves) && narrow_cloud(w[1], w[3], octaves) ? 0u : 1u;
      }
    }
  }
}

// Round-to-nearest (ties away) onto the 10-bit TF32 mantissa with two integer operations; the conversion
// instruction shares the quarter-rate pipe with ex2, which the weights already saturate. Works on the
// magnitude, so it is valid for either sign; the inputs here are finite weights in [0, ~1].
__device__ __forceinline__ float round_tf32_pos(float w) {
  return __uint_as_float((__float_as_uint(w) + 0x1000u) & 0xffffe000u);
}

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
        "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
        "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])), "r"(__float_as_uint(v[8])),
        "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
        "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])),
        "r"(__float_as_uint(v[15])), "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])),
        "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])), "r"(__float_as_uint(v[20])),
        "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
        "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])),
        "r"(__float_as_uint(v[27])), "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])),
        "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
      : "memory");
}

}  // namespace
}  // namespace tc
}  // namespace fs
