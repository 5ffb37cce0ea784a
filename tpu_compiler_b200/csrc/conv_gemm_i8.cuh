// INT8 implicit-GEMM convolution / fully-connected kernel for sm_100a.
//
// Replaces, for INT8 graphs, the reference's Conv2DOpKernel::invoke
// (lib/Dialect/TPU/Interpreter/core/conv.cpp:80-104: fp32 MKL-DNN convolution on
// integer-valued floats followed by quantizeActivationInt8PerChannelMultiplierAndRShift,
// lib/Dialect/TPU/Quantization/QuantizationArithmetic.cpp:849-871) and
// FullyConnectedOpKernel::invoke (core/fullyconnected.cpp:44-91).
//
// The product is computed transposed, D[128 output channels][128 output pixels]: the weight
// tile ([Cout][tap][Cin] int8, 3-D tiled TMA load) is the tensor core's A operand and the
// activation tile its B operand, fetched either by an im2col-mode TMA load (any kh/kw/
// stride/dilation/padding; out-of-image taps arrive as zeros) or by a plain 2-D tiled TMA
// load (1x1 stride-1 convolutions, fully-connected, pre-expanded patch matrices). Tiles land
// in shared memory in the 32/64/128-byte swizzled K-major layout the tensor core reads and
// accumulate in int32 in tensor memory (tcgen05.mma kind::i8). With channels on the TMEM
// lanes every epilogue thread owns ONE output channel, so its bias / multiplier / rshift
// constants sit in registers instead of being re-read per value; the epilogue requantises,
// saturates, applies ReLU, transposes through shared memory with transposing matrix stores, and
// stores 8 channels of one pixel per lane (a warp writes whole 32-byte sectors of the NHWC output).
//
// Warp roles (320 threads): warp 0 = TMA producer, warp 1 = TMEM owner + MMA
// issuer, warps 2..9 = epilogue (two warps per TMEM lane quarter, alternating
// 32-column groups).
// Every wait is bounded: on expiry the CTA records an error code in p.err and
// leaves through the common tear-down (TMEM freed, in-flight copies drained).
#pragma once
#include "common.cuh"
#include <type_traits>
#include <cuda.h>

namespace tpucb {

struct ConvGemmParams {
  int M_total;    // rows of the implicit GEMM: N*OH*OW (or m for fully-connected)
  int OH, OW;     // output spatial size (im2col mode)
  int sh, sw;     // stride
  int pt, pl;     // top / left padding
  int dh, dw;     // dilation
  int kh, kw;     // filter size (taps = kh*kw; 1 in tiled mode)
  int c_chunks;   // ceil(Cin_pad / BK)
  int BK;         // K bytes per pipeline stage: 32, 64 or 128 (= swizzle span)
  int m_tile;     // pixels per tile: 256 in dual mode, else 128 or 64 = the tensor core's N
  int BN;         // channel tile = tensor-core M, always 128 (rows past n_valid are zero-filled)
  int n_valid;    // number of valid (padded) output channels
  int ldc;        // output row pitch in bytes
  int c_off;      // first output channel written inside a row
  int stages;     // pipeline depth
  int dual;       // 1: at most 64 channels: two 128-pixel sub-tiles share the 128 TMEM lanes (see kernel)
  int w_resident; // 1: the CTA keeps all K blocks of its channel tile's weights in shared memory
  int a_mode;     // 0: A is a 2-D [M][K] matrix, 1: im2col TMA
  int ksteps;     // MMAs (32 bytes of K) per K block: BK / 32, fewer when the block's tail is padding
  // Pixel groups (WindowPlan): > 1 means that a row of the implicit GEMM is `group` neighbouring output pixels, whose
  // channels are 128 / group apart on the TMEM lanes; M_total, OW and ldc then count groups, ldc_px is one pixel's pitch.
  int group, ldc_px;
  int act;        // 0 none, 1 ReLU, 2 leaky (non-QDM pos/neg rescale of the int8 result),
                  // 3 the eltwise add that consumes this convolution, with the residual tensor `res` (see add_*)
  int tmem_cols;  // 256: two accumulator buffers of 128 pixel columns
  int leaky_mp, leaky_rp, leaky_mn, leaky_rn;
  uint32_t idesc; // tcgen05 instruction descriptor
  const int32_t *bias;   // [n_valid]
  const int32_t *mult;   // [n_valid]
  const int32_t *rshift; // [n_valid]
  const FloatRequant *fq; // [n_valid], or null: the floating-point form of the requantisation does not apply
  int8_t *out;
  int fastq;      // bit 0: the multiply-high form of the requantisation applies (requant_fast; set by the host);
                  // bit 1: every rshift of the layer is >= 1
  int8_t *out2;   // act == 2 / 3: the activation (or sum) goes here and `out` keeps the plain convolution result
  // act == 3 (EltwiseAddOpKernel::i8_invoke, core/eltwise.cpp:52-85, applied to this convolution's int8 result x and the
  // tensor `res` of the same geometry): sat8(relu?((x * add_ms + res * add_mr + 2^(add_r - 1)) >> add_r))
  const int8_t *res;
  int add_ms, add_mr, add_r, add_relu;
  int *err;       // device error word (0 = ok)
  // Self-test of the bounded waits (interpreter option "selftest_lost_arrival"): wait_rounds > 0 shortens every wait of
  // this launch to that many rounds of 1024 polls, and with lose_arrival the epilogue warps never hand an accumulator
  // buffer back, so that the MMA issuer's wait for it runs out and the launch ends through its error path (status
  // kErrAccWait) with no copy in flight. 0 / 0 in every ordinary launch.
  int wait_rounds, lose_arrival;
  // Split K (launches with fewer tiles than CTA slots and a long K, e.g. every layer of the last two stages at batch
  // 1): split_k > 1 CTAs share a tile, each takes k_per K blocks, adds its int32 partial accumulator to `ws`
  // ([tile][pixel column][channel lane], zero between launches) with red.global.add and counts itself in `ws_count`;
  // the CTA whose count completes the tile (no CTA waits for another) reads the sums back, runs the ordinary epilogue
  // on them and leaves `ws` and the counter zero again. Plain tiles only (not dual, INT8).
  int split_k, k_per;
  int32_t *ws;
  unsigned int *ws_count;
};

namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// True in one lane of a converged warp. The compiler knows that a branch on it holds one thread: copies and MMAs, whose
// operands are registers of the whole warp, are then issued once, not in a loop over the lanes that might be active (with
// `lane == 0` instead: ResNet-50 INT8 batch 1 283 us against 259, batch 19 442 against 422, fp32 batch 64 5796 against 5641).
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
  return ok != 0;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
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
// The same with a suspend-time hint (nanoseconds): the thread may sleep in the instruction until the phase completes
// or that much time has passed, instead of coming back after the (short) default limit; a waiting role then spends
// few issue slots on its polling loop.
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
// Bounded wait: returns false when the barrier did not flip within the limit.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity,
                                                  volatile int *abort_flag, int rounds = 1024) {
  // `rounds` (1024 by default) rounds of 1024 polls of at most a microsecond each (about a second in all): the abort
  // flag (another role of this CTA gave up) is read once per round
  for (int round = 0; round < rounds; ++round) {
#pragma unroll 1
    for (int it = 1024; it > 0; --it)
      if (mbar_try_wait_hint(bar, parity, 1000u)) return true;
    if (*abort_flag) return false;
  }
  return false;
}
// The same by a whole warp, whose lanes get one answer: the loops of the copying and issuing warps are then uniform, and what
// they compute stays in the registers that the copies and MMAs take (by one lane of a branch, every operand was moved there
// for every instruction: batch 1 259 -> 248 us, batch 19 422 -> 401, fp32 5641 -> 5487).
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag, int rounds) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, abort_flag, rounds));
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void *tmap, uint32_t bar, int x,
                                            int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(tmap), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const void *tmap, uint32_t bar, int x,
                                            int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_load_im2col_4d(uint32_t dst, const void *tmap, uint32_t bar,
                                                   int c, int w, int h, int n, uint16_t off_w,
                                                   uint16_t off_h) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};" ::"r"(dst),
      "l"(tmap), "r"(bar), "r"(c), "r"(w), "r"(h), "r"(n), "h"(off_w), "h"(off_h)
      : "memory");
}
__device__ __forceinline__ void tcgen05_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tcgen05_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tcgen05_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tcgen05_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tcgen05_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   bar)
               : "memory");
}
__device__ __forceinline__ void tcgen05_mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                               uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same MMA with the descriptors given as 32-bit halves (only the low words change between
// K steps and stages) and, when ACCUMULATE, a constant-true accumulate predicate: the issuing
// thread's loop carries no 64-bit arithmetic.
template <bool ACCUMULATE>
__device__ __forceinline__ void tcgen05_mma_i8_lohi(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo,
                                                    uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  if (ACCUMULATE) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "setp.eq.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}
// kind::f16 with BF16 operands and fp32 accumulation (BF16 graphs): 16 elements = 32 bytes of K per MMA
template <bool ACCUMULATE>
__device__ __forceinline__ void tcgen05_mma_f16_lohi(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo,
                                                     uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  if (ACCUMULATE) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "setp.eq.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}
// kind::tf32 with fp32 words as operands (their low 13 mantissa bits do not take part) and fp32 accumulation:
// 8 elements = 32 bytes of K per MMA
template <bool ACCUMULATE>
__device__ __forceinline__ void tcgen05_mma_tf32_lohi(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo,
                                                      uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  if (ACCUMULATE) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "setp.eq.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}
// KSTEPS MMAs of one K block (32 bytes of K each: +2 in the descriptors' 16-byte address units).
// KIND: 0 kind::i8, 1 kind::f16 on BF16 operands, 2 kind::tf32
template <int KSTEPS, int KIND = 0>
__device__ __forceinline__ void tcgen05_mma_i8_kblock(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi,
                                                      uint32_t idesc, uint32_t accumulate_first) {
  if (KIND == 2) tcgen05_mma_tf32_lohi<false>(d_tmem, a_lo, hi, b_lo, hi, idesc, accumulate_first);
  else if (KIND == 1) tcgen05_mma_f16_lohi<false>(d_tmem, a_lo, hi, b_lo, hi, idesc, accumulate_first);
  else tcgen05_mma_i8_lohi<false>(d_tmem, a_lo, hi, b_lo, hi, idesc, accumulate_first);
#pragma unroll
  for (int k = 1; k < KSTEPS; ++k) {
    if (KIND == 2) tcgen05_mma_tf32_lohi<true>(d_tmem, a_lo + 2 * k, hi, b_lo + 2 * k, hi, idesc, 1u);
    else if (KIND == 1) tcgen05_mma_f16_lohi<true>(d_tmem, a_lo + 2 * k, hi, b_lo + 2 * k, hi, idesc, 1u);
    else tcgen05_mma_i8_lohi<true>(d_tmem, a_lo + 2 * k, hi, b_lo + 2 * k, hi, idesc, 1u);
  }
}
__device__ __forceinline__ void tcgen05_ld_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tcgen05_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

} // namespace ptx

// Shared-memory matrix descriptor for a K-major tile whose rows are `BK` bytes
// long and swizzled over `BK` bytes (BK in {32,64,128}): 8-row groups are
// 8*BK bytes apart (stride byte offset); the leading byte offset is unused for
// swizzled K-major tiles; bits 46-47 carry the sm_100 descriptor version.
__device__ __forceinline__ uint64_t make_kmajor_desc(uint32_t smem_addr, int BK) {
  uint64_t layout = BK == 128 ? 2ull : (BK == 64 ? 4ull : 6ull);
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3ffffu) >> 4);
  d |= (uint64_t)1 << 16;                            // leading byte offset (ignored)
  d |= (uint64_t)(((uint32_t)(8 * BK)) >> 4) << 32;  // stride byte offset
  d |= (uint64_t)1 << 46;                            // descriptor version (Blackwell)
  d |= layout << 61;
  return d;
}

constexpr int kEpilogueWarps = 8;
constexpr int kConvThreads = 64 + 32 * kEpilogueWarps;
constexpr int kMaxStages = 8;
constexpr int kSmemHeader = 1024 + 8 * 1024; // barriers, then kStageBytes for each epilogue warp

// Records why a launch gave up, in the device word that later CTAs and kernels look at and in the host's own memory, whose
// address stands 8 bytes behind the device word (ErrWord).
__device__ __forceinline__ void report_error(int *err, int code) {
  atomicExch(err, code);
  int *host = *reinterpret_cast<int **>(err + 2);
  *reinterpret_cast<volatile int *>(host) = code;
  __threadfence_system();
}

enum ConvErr { kErrFullWait = 1, kErrEmptyWait = 2, kErrAccWait = 3 };

// A warp's wait has run out: the host is told, unless another role of the CTA has done so, and then the other roles. (The flag is
// raised behind the read by the lane that reports: a lane that came first would have hidden the error.)
__device__ __forceinline__ void wait_expired(int *err, volatile int *abort_flag, int code) {
  if ((threadIdx.x & 31) == 0 && !*abort_flag) report_error(err, code);
  __syncwarp();
  *abort_flag = 1;
}

// Per-channel requantisation constants, held in registers by the thread that owns the channel.
// The reference computes, for s = acc + bias and multiplier M in [0, 2^31),
//   hi = SaturatingRoundingDoublingHighMul(s, M) = floor((s * M + 2^30) / 2^31)
//        (adding 2^30 and flooring equals its sign-dependent nudge followed by a division that
//        truncates toward zero, for either sign),
//   q  = RoundingDivideByPOT(hi, r) = (hi + rnd - [hi < 0 and r > 0]) >> r, rnd = 2^(r-1) (0 if r = 0),
// then saturates (and ReLU clamps at 0, so there rnd is folded into the constant and the sign term
// dropped). requant_one forms the product once, unsigned and doubled, so that hi is simply the HIGH
// WORD of one 32 x 32 + 64 multiply-add:
//   s' = s + 2^31 (offset binary, one add of `sbias` = bias + 2^31), M2 = 2 * M (fits unsigned 32),
//   2 * (s * M + C) = s' * M2 + (2 * C - 2^31 * M2)   (mod 2^64),  C = 2^30 (+ rnd * 2^31 with ReLU),
//   hi = that >> 32.
struct ChanConst {
  uint32_t M2, sbias;
  int32_t r, rnd, s1; // s1 = 31 when r > 0, 32 when r == 0: (uint)hi >> s1 is the "negative and r > 0" bit
  unsigned long long c2;
  uint32_t kc;        // multiply-high form only (requant_fast), where r holds r + 1
  int32_t r0mask;     // multiply-high form: -1 when r == 0 (no sign term for this channel), else 0
};

__device__ __forceinline__ ChanConst load_chan_const(const ConvGemmParams &p, int n) {
  ChanConst c;
  const bool v = n < p.n_valid;
  const int32_t M = v ? p.mult[n] : 0;
  const int32_t b = v ? p.bias[n] : 0;
  c.r = v ? p.rshift[n] : 0;
  const unsigned long long rnd = c.r > 0 ? (1ull << (c.r - 1)) : 0ull;
  unsigned long long C = 1ull << 30;
  if (p.act == 1) C += rnd << 31;
  c.M2 = (uint32_t)M << 1;
  c.c2 = 2ull * C - ((unsigned long long)c.M2 << 31);
  c.sbias = (uint32_t)b + 0x80000000u;
  c.rnd = (int32_t)rnd;
  c.s1 = c.r > 0 ? 31 : 32;
  c.kc = 0;
  c.r0mask = c.r == 0 ? -1 : 0;
  if (p.fastq & 1) {
    // multiply-high form: see requant_fast
    const uint32_t k = 1u + 2u * (uint32_t)rnd;
    c.sbias = 2u * (uint32_t)b + 0x80000000u;
    // the sign term costs 2 when s < 0: the constant carries the -2 and the kernel gives it back when s >= 0
    c.kc = p.act == 1 ? k - (uint32_t)M : k - (uint32_t)M - (c.r > 0 ? 2u : 0u);
    c.r = c.r + 1;
    if (!v) { // a lane past the layer's channels: s2 = 0, no sign term, result 0
      c.sbias = 0u;
      c.kc = 0u;
    }
  }
  return c;
}

// One requantised value BEFORE the final int8 saturation (pack4_sat applies it).
template <int ACT>
__device__ __forceinline__ int requant_one(int32_t acc, const ChanConst &q, const ConvGemmParams &p) {
  unsigned long long x;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(x) : "r"((uint32_t)acc + q.sbias), "r"(q.M2), "l"(q.c2));
  const int32_t hi = (int32_t)(uint32_t)(x >> 32);
  if (ACT == 1) {
    return max(hi, 0) >> q.r; // rnd already folded into c2; the upper clamp happens in the pack
  }
  uint32_t adj;
  asm("shr.u32 %0, %1, %2;" : "=r"(adj) : "r"((uint32_t)hi), "r"((uint32_t)q.s1)); // shifts >= 32 give 0
  int v = (hi + q.rnd - (int)adj) >> q.r;
  if (ACT == 2) v = min(max(v, -128), 127); // the leaky rescale below works on the saturated int8 value
  return v;
}
// The same value from ONE multiply-high. With t = floor(s * M / 2^30), hi = floor((t + 1) / 2) and, nesting the
// floors, q = floor((t + k - 2 * neg) / 2^(r + 1)), k = 1 + 2 * rnd, neg = [hi < 0 and r > 0].
//   Offset binary: s2 = 2 * (s + 2^30) is a non-negative 32-bit number whose top bit says s >= 0, and
//   mulhi(s2, 2M) = t + M exactly, so the addend kc = k - M gives t + k.
//   ReLU (ACT 1): no sign term. For s >= 0 the value is (t + k) >> (r + 1); for s < 0 it is <= 0 ((t + k) < 2^(r + 1)
//         there), which the caller clamps to 0 on the packed bytes (relu4): no clamp per value.
//   else: neg may be replaced by [s < 0 and r > 0]: the two differ only for t = -1 (hi = 0), where both forms
//         give 0. With m = s2 >> 31 (arithmetic: -1 for s >= 0, 0 for s < 0) the term is -2 - 2m; the -2 sits in kc.
//         R1 = every channel of the layer has r > 0; otherwise the channels with r = 0 switch the term off (r0mask).
// Valid for |s| < 2^29 and r <= 29 (no 32-bit overflow); the host sets fastq only when every channel of the
// layer and the largest possible |acc| satisfy that, else requant_one runs.
template <int ACT, bool R1>
__device__ __forceinline__ int requant_fast(int32_t acc, const ChanConst &q, const ConvGemmParams &p) {
  // The instructions are spelled out. Measured rates on this SM, lanes per clock: add / min / max 127; shifts, logic,
  // permutes, saturating packs and 32-bit multiply-adds 64, the last on a pipe of their own; multiply-high and
  // shuffles 32; the 64-bit multiply-add 16. The doubling and the sign term are multiply-adds, which run beside the
  // two shifts on the ALU: 122 -> 112 us on a 64 -> 256 channel 1x1 layer at batch 256; written as adds instead,
  // both 123 us, the doubling alone 111, the sign term alone 114.
  uint32_t s2, tk;
  asm("mad.lo.u32 %0, %1, 2, %2;" : "=r"(s2) : "r"((uint32_t)acc), "r"(q.sbias));
  asm("mad.hi.u32 %0, %1, %2, %3;" : "=r"(tk) : "r"(s2), "r"(q.M2), "r"(q.kc));
  int32_t v;
  if (ACT == 1) {
    asm("shr.s32 %0, %1, %2;" : "=r"(v) : "r"((int32_t)tk), "r"((uint32_t)q.r));
    return v;
  }
  int32_t m, x;
  asm("shr.s32 %0, %1, 31;" : "=r"(m) : "r"((int32_t)s2));
  if (!R1) m &= ~q.r0mask; // r == 0: kc carries no -2 and nothing is given back
  asm("mad.lo.s32 %0, %1, -2, %2;" : "=r"(x) : "r"(m), "r"((int32_t)tk));
  asm("shr.s32 %0, %1, %2;" : "=r"(v) : "r"(x), "r"((uint32_t)q.r));
  if (ACT == 2) v = min(max(v, -128), 127);
  return v;
}
// The INT8 eltwise add of four packed convolution results x with four packed residual values y: (x * ms + y * mr + rnd) >> r
// per byte through one four-way dot product each, whose multipliers pick one of the two pairs in a word; saturated, ReLU on the
// packed bytes. (Two-way dot products with 16-bit multipliers, scaled so that the results are upper bytes, need no shifts and
// are slower: ResNet-50 batch 256 2158 us against 2113, 64 620 against 604.)
struct AddConsts {
  int m01, m23, rnd, r; // (ms, mr, 0, 0) and (0, 0, ms, mr) as bytes
  bool relu;
};
__device__ __forceinline__ AddConsts make_add_consts(const ConvGemmParams &p) {
  AddConsts c;
  c.m01 = (int)((uint32_t)(uint8_t)p.add_ms | ((uint32_t)(uint8_t)p.add_mr << 8));
  c.m23 = (int)((uint32_t)c.m01 << 16);
  c.rnd = p.add_r > 0 ? (1 << (p.add_r - 1)) : 0;
  c.r = p.add_r;
  c.relu = p.add_relu != 0;
  return c;
}
__device__ __forceinline__ uint32_t add4_packed(uint32_t x, uint32_t y, const AddConsts &c) {
  const int a = (int)__byte_perm(x, y, 0x5140), b = (int)__byte_perm(x, y, 0x7362); // (x0, y0, x1, y1), (x2, y2, x3, y3)
  const uint32_t w = pack4_sat(__dp4a(a, c.m01, c.rnd) >> c.r, __dp4a(a, c.m23, c.rnd) >> c.r, __dp4a(b, c.m01, c.rnd) >> c.r,
                               __dp4a(b, c.m23, c.rnd) >> c.r);
  return c.relu ? relu_bytes(w) : w;
}
// INT8 leaky ReLU of four packed convolution results (core/activation.cpp:126-153): (v * m + rnd) >> r with the multiplier of
// the value's sign, positive values unchanged where their multiplier is 0; the pack saturates.
__device__ __forceinline__ uint32_t leaky4(uint32_t w, const ConvGemmParams &p) {
  const int rp = p.leaky_mp != 0 ? p.leaky_rp : 0, rn = p.leaky_rn;
  const int ap = rp > 0 ? 1 << (rp - 1) : 0, an = rn > 0 ? 1 << (rn - 1) : 0, mp = p.leaky_mp != 0 ? p.leaky_mp : 1, mn = p.leaky_mn;
  auto one = [&](int v) {
    const bool pos = v > 0;
    return (v * (pos ? mp : mn) + (pos ? ap : an)) >> (pos ? rp : rn);
  };
  auto below = [&](int v) { return v > 0 ? v : (v * mn + an) >> rn; };
  if (p.leaky_mp != 0) return pack4_sat(one(sext_byte<0>(w)), one(sext_byte<1>(w)), one(sext_byte<2>(w)), one(sext_byte<3>(w)));
  return pack4_sat(below(sext_byte<0>(w)), below(sext_byte<1>(w)), below(sext_byte<2>(w)), below(sext_byte<3>(w)));
}

// Channel of a 32-channel block that sits on TMEM lane `lane` of its quarter, and the row of the packed weights that puts it
// there. Lanes 4i + j hold channels 8j + i: the transposing matrix store below then leaves runs of eight channels.
TPUCB_HD int lane_channel(int lane) { return 8 * (lane & 3) + (lane >> 2); }
TPUCB_HD int packed_row(int channel) { return (channel & ~31) | (4 * (channel & 7) + ((channel & 31) >> 3)); }

// A warp's kStageBytes of shared memory, through which the epilogue turns "one channel, several pixels" per lane into "one
// pixel, eight channels": matrix stores that transpose (rows of 16 bytes, `put` is this lane's), 16-byte loads from `get`.
// Per 32 channels x 32 pixels two stores and two loads (INT8); exchanged between lanes by shuffles and byte permutes it was
// 32 instructions, and 16 for the stores and their addresses instead of 8. ResNet-50, us alone before and after: INT8 batch 256
// 2555 -> 2470 (64 -> 256 channels, 1x1, 56 x 56: 82 -> 76), batch 19 465 -> 442; BF16 batch 128 2459 -> 2276 (72 -> 47).
constexpr int kStageBytes = 1024;
struct StageLane {
  uint32_t put, get;
  int px; // the first pixel that this lane gets
};
// PX_PER_WORD: pixels that a lane packs into one word before the transposition (4 of one byte, 2 of two)
template <int PX_PER_WORD> __device__ __forceinline__ StageLane make_stage_lane(uint32_t warp_stage, int lane) {
  const int pair = lane >> 3, h = (lane >> 2) & 1;
  return StageLane{warp_stage + lane * 16, warp_stage + pair * 128 + (2 * (lane & 3) + h) * 16, (PX_PER_WORD * pair) + h};
}
__device__ __forceinline__ void lds128(uint32_t at, uint32_t (&v)[4]) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(at) : "memory");
}
// INT8. In: byte b of w[k] is pixel 4k + b of this lane's channel. Out: u[2i], u[2i + 1] hold channels 8 (lane & 3) .. + 7 of
// pixel st.px + stage_step8(i).
__device__ __forceinline__ constexpr int stage_step8(int i) { return 2 * (i & 1) + 16 * (i >> 1); }
__device__ __forceinline__ void transpose_i8(const uint32_t (&w)[8], uint32_t (&u)[8], const StageLane &st) {
  __syncwarp(); // the previous chunk has been read
  asm volatile("stmatrix.sync.aligned.m16n8.x4.trans.shared.b8 [%0], {%1, %2, %3, %4};" ::"r"(st.put), "r"(w[0]), "r"(w[1]), "r"(w[2]),
               "r"(w[3]) : "memory");
  asm volatile("stmatrix.sync.aligned.m16n8.x4.trans.shared.b8 [%0], {%1, %2, %3, %4};" ::"r"(st.put + 512u), "r"(w[4]), "r"(w[5]),
               "r"(w[6]), "r"(w[7]) : "memory");
  __syncwarp();
  uint32_t a[4], b[4];
  lds128(st.get, a);
  lds128(st.get + 512u, b);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    u[i] = a[i];
    u[4 + i] = b[i];
  }
}
// address of pixel `px` from `base`, by one wide multiply-add (the multiply-add pipe has room, the integer ALU has not)
__device__ __forceinline__ unsigned long long px_addr(const void *base, int px, int pitch) {
  unsigned long long a;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(a) : "r"((uint32_t)px), "r"((uint32_t)pitch), "l"((unsigned long long)base));
  return a;
}
__device__ __forceinline__ void stg64(unsigned long long at, uint32_t x, uint32_t y) {
  asm volatile("st.global.v2.b32 [%0], {%1, %2};" ::"l"(at), "r"(x), "r"(y) : "memory");
}

// Epilogue of one accumulator buffer for the 32 channels (TMEM lanes) of this warp.
//   lane_addr  TMEM address of the warp's lane quarter in the buffer
//   out8       output address of (pixel m0, this lane's group of eight channels)
//   ch8_ok     that group lies inside the valid channels
//   ncols      pixel columns of the accumulator buffer that the tile fills (128, or 64 for half tiles)
//   FORM       of the requantisation: 0 requant_one, 1 requant_fast, 2 requant_fast with every rshift >= 1, 3 float_requant4
template <int ACT, int FORM, bool FROM_WS = false, class Consts = ChanConst>
__device__ __forceinline__ void epilogue_channels_impl(const ConvGemmParams &p, uint32_t lane_addr, int8_t *out8,
                                                       bool ch8_ok, int m0, int half, int halves, int lane,
                                                       const Consts &cc, const FloatRequantShared &fs, const StageLane &st, int ncols,
                                                       int32_t *ws_lane = nullptr) {
  constexpr int QACT = ACT == 3 ? 0 : ACT; // the fused add works on the plain (no activation) int8 result
  // four pixels of this lane's channel, packed
  auto rq4 = [&](uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) -> uint32_t {
    if constexpr (FORM == 3) {
      return float_requant4<QACT == 1>(a0, a1, a2, a3, cc, fs);
    } else {
      auto rq = [&](uint32_t a) {
        if constexpr (FORM == 0) return requant_one<QACT>((int32_t)a, cc, p);
        else return requant_fast<QACT, FORM == 2>((int32_t)a, cc, p);
      };
      const uint32_t w = pack4_sat(rq(a0), rq(a1), rq(a2), rq(a3));
      return FORM != 0 && ACT == 1 ? relu_bytes(w) : w; // the multiply-high form leaves the ReLU clamp to the packed bytes
    }
  };
  // (Software-pipelining these loads in 16-column pieces made the epilogue alone 14% faster and the whole
  // kernel 4% slower, so the two loads of a chunk are simply issued together.)
  const int cols = min(ncols, p.M_total - m0);
  int left = ch8_ok ? p.M_total - m0 - half * 32 - st.px : 0; // pixels in range from this lane's first one of the chunk
  unsigned long long o = px_addr(out8, half * 32 + st.px, p.ldc);
  for (int colg = half * 32; colg < cols; colg += 32 * halves, left -= 32 * halves, o = px_addr((const void *)o, 32 * halves, p.ldc)) {
    uint2 y[4];
    if (ACT == 3) {
      // the residual words of the fused eltwise add sit where the results go (same geometry): fetched first, so
      // that their latency passes under the accumulator loads and the requantisation
      const int8_t *rp = p.res + (o - (unsigned long long)p.out);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        y[i] = make_uint2(0u, 0u);
        if (stage_step8(i) < left) y[i] = __ldg(reinterpret_cast<const uint2 *>(rp + (size_t)stage_step8(i) * p.ldc));
      }
    }
    uint32_t acc0[16], acc1[16];
    if (FROM_WS) {
      // split K: the summed accumulators of all the tile's CTAs, [pixel column][128 channel lanes] in global memory;
      // read past L1 (other SMs wrote them) and left zero for the next launch
      int32_t *src = ws_lane + (size_t)colg * 128;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        acc0[k] = (uint32_t)__ldcg(src + (size_t)k * 128);
        acc1[k] = (uint32_t)__ldcg(src + (size_t)(16 + k) * 128);
      }
#pragma unroll
      for (int k = 0; k < 32; ++k) __stcg(src + (size_t)k * 128, 0);
    } else {
      ptx::tcgen05_ld_x16(lane_addr + (uint32_t)colg, acc0);
      ptx::tcgen05_ld_x16(lane_addr + (uint32_t)colg + 16u, acc1);
      ptx::tcgen05_wait_ld();
    }
    uint32_t w[8], u[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      w[k] = rq4(acc0[4 * k + 0], acc0[4 * k + 1], acc0[4 * k + 2], acc0[4 * k + 3]);
      w[4 + k] = rq4(acc1[4 * k + 0], acc1[4 * k + 1], acc1[4 * k + 2], acc1[4 * k + 3]);
    }
    transpose_i8(w, u, st);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (stage_step8(i) >= left) continue;
      const unsigned long long at = px_addr((const void *)o, stage_step8(i), p.ldc);
      const uint32_t a = u[2 * i], b = u[2 * i + 1];
      if (ACT == 3) {
        // fused eltwise add: both tensors are written
        const AddConsts ac = make_add_consts(p);
        stg64(at, a, b);
        stg64(at + (unsigned long long)(p.out2 - p.out), add4_packed(a, y[i].x, ac), add4_packed(b, y[i].y, ac));
      } else if (ACT == 2) {
        // fused leaky ReLU: the activation works on the packed, saturated values (eight channels of one pixel); the plain
        // result goes to `out` when the graph keeps that tensor
        if (p.out2) stg64(at, a, b);
        stg64(p.out2 ? at + (unsigned long long)(p.out2 - p.out) : at, leaky4(a, p), leaky4(b, p));
      } else {
        stg64(at, a, b);
      }
    }
  }
}

// The same with the fused eltwise add and the floating-point requantisation, for the two 32-pixel chunks of a warp. With three
// tensors in every chunk the accesses to memory count: the four warps that hold the channels of the same pixels exchange their
// results through shared memory, and each handles 8 pixels x 128 channels, 16 bytes a lane, four pixels per access (of its own 32
// channels it was 8 bytes a lane and 8 pixels, twice the accesses of twice the lines each, and the
// load/store pipe 60% busy: ResNet-50 batch 256 2336 us against 2210, with three modules in flight 2127 / 2003, batch 64 605 / 573).
// The residual words are fetched a chunk ahead, across tiles: those of the first chunk during the tile before (`y`), those of the
// second while the first is worked on. Fetched where they are needed, they cost a memory latency per chunk.
struct AddLane {
  uint32_t put, get; // this lane's row of its warp's matrix stores; its 8 channels in the exchange, the next 8 are 32 bytes on
  int px, ch;        // its first pixel of a chunk (the second is 4 on) and its first channel of a tile
};
constexpr int kAddQuarter = kStageBytes + 32; // 32 bytes more: a lane group's eight accesses meet in a bank two by two, not four by four
__device__ __forceinline__ AddLane make_add_lane(uint32_t stage, int half, int quarter, int lane) {
  const uint32_t at = stage + (uint32_t)(half * 4 * kAddQuarter);
  const int c16 = lane & 7, h = (lane >> 3) & 1, pos = lane >> 4;
  return AddLane{at + (uint32_t)(quarter * kAddQuarter + lane * 16),
                 at + (uint32_t)((c16 >> 1) * kAddQuarter + (quarter >> 1) * 512 + (quarter & 1) * 256 + (4 * (c16 & 1) + h) * 16 + pos * 8),
                 8 * quarter + (lane >> 3), 16 * c16};
}
// The same for BF16, sixteen pixels at a time: 4 pixels x 128 channels per warp, two pixels per access (the second is 2 on).
// ResNet-50 batch 128 2160 -> 2088 us, with three modules in flight 1862 -> 1791, batch 32 802 / 542 -> 776 / 525.
constexpr int kAddQuarter16 = kStageBytes + 16;
__device__ __forceinline__ AddLane make_add_lane16(uint32_t stage, int half, int quarter, int lane) {
  const uint32_t at = stage + (uint32_t)(half * 4 * kAddQuarter16);
  const int c16 = lane & 15, h = lane >> 4;
  return AddLane{at + (uint32_t)(quarter * kAddQuarter16 + lane * 16),
                 at + (uint32_t)((c16 >> 2) * kAddQuarter16 + (quarter >> 1) * 512 + (quarter & 1) * 256 + (2 * (c16 & 3) + h) * 16),
                 4 * quarter + h, 8 * c16};
}
// `at`: this lane's first pixel of the chunk; left: pixels in range from there (0: the lane has no channels)
__device__ __forceinline__ void fetch_residual(uint4 (&y)[2], const int8_t *at, int left, int pitch) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (4 * i < left)
      asm volatile("ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(y[i].x), "=r"(y[i].y), "=r"(y[i].z), "=r"(y[i].w) : "l"(px_addr(at, 4 * i, pitch)));
}
// out16: this lane's first pixel of the tile; mine: the warp's accumulators hold channels of the layer
__device__ __forceinline__ void epilogue_add_fq(const ConvGemmParams &p, uint32_t lane_addr, int8_t *out16, int left, bool mine, int m0, int half,
                                                const FloatRequantPairs<false> &q, const FloatRequantShared &fs, const AddLane &al, int ncols,
                                                uint4 (&y)[2], const int8_t *next, int next_left) {
  const int col0 = half * 32, col1 = col0 + 64;
  const AddConsts ac = make_add_consts(p);
  const unsigned long long to_sum = (unsigned long long)(p.out2 - p.out);
  auto meet = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory"); };
  auto chunk = [&](int colg, const uint4 (&res)[2]) {
    uint32_t w[8];
    if (mine) {
      uint32_t acc0[16], acc1[16];
      ptx::tcgen05_ld_x16(lane_addr + (uint32_t)colg, acc0);
      ptx::tcgen05_ld_x16(lane_addr + (uint32_t)colg + 16u, acc1);
      ptx::tcgen05_wait_ld();
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        w[k] = float_requant4<false>(acc0[4 * k + 0], acc0[4 * k + 1], acc0[4 * k + 2], acc0[4 * k + 3], q, fs);
        w[4 + k] = float_requant4<false>(acc1[4 * k + 0], acc1[4 * k + 1], acc1[4 * k + 2], acc1[4 * k + 3], q, fs);
      }
    }
    meet(); // the chunk before has been read
    if (mine) {
      asm volatile("stmatrix.sync.aligned.m16n8.x4.trans.shared.b8 [%0], {%1, %2, %3, %4};" ::"r"(al.put), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                   "r"(w[3]) : "memory");
      asm volatile("stmatrix.sync.aligned.m16n8.x4.trans.shared.b8 [%0], {%1, %2, %3, %4};" ::"r"(al.put + 512u), "r"(w[4]), "r"(w[5]),
                   "r"(w[6]), "r"(w[7]) : "memory");
    }
    meet();
    const unsigned long long o = px_addr(out16, colg, p.ldc);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t u[4];
      asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(u[0]), "=r"(u[1]) : "r"(al.get + 128u * i) : "memory");
      asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(u[2]), "=r"(u[3]) : "r"(al.get + 128u * i + 32u) : "memory");
      if (4 * i < left - colg) {
        const unsigned long long at = px_addr((const void *)o, 4 * i, p.ldc);
        asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(at), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]) : "memory");
        asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(at + to_sum), "r"(add4_packed(u[0], res[i].x, ac)),
                     "r"(add4_packed(u[1], res[i].y, ac)), "r"(add4_packed(u[2], res[i].z, ac)), "r"(add4_packed(u[3], res[i].w, ac)) : "memory");
      }
    }
  };
  uint4 y1[2];
  const bool two = col1 < ncols && m0 + col1 < p.M_total;
  if (two) fetch_residual(y1, p.res + (out16 - p.out) + (size_t)col1 * p.ldc, left - col1, p.ldc);
  if (col0 < ncols && m0 + col0 < p.M_total) chunk(col0, y);
  fetch_residual(y, next + (size_t)col0 * p.ldc, next_left - col0, p.ldc);
  if (two) chunk(col1, y1);
}

// Two BF16 roundings (and ReLU) by the hardware; a multiply-add by zero carries every result that it made infinite or NaN into
// `odd`, and a caller that finds one there rounds again by the reference's bit rule (bf16_pack_rule).
template <bool RELU> __device__ __forceinline__ uint32_t bf16_pack_relu(unsigned long long v, uint32_t &odd) {
  float lo, hi;
  uint32_t w;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  if (RELU) asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(hi), "f"(lo));
  else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(hi), "f"(lo));
  asm("fma.rn.bf16x2 %0, %1, %2, %0;" : "+r"(odd) : "r"(w), "r"(0u));
  return w;
}
template <bool RELU> __device__ __forceinline__ uint32_t bf16_pack_rule(uint32_t a0, uint32_t a1, float bias) {
  float lo = __fadd_rn(bits_f32(a0), bias), hi = __fadd_rn(bits_f32(a1), bias);
  if (RELU) {
    lo = lo > 0.0f ? lo : 0.0f;
    hi = hi > 0.0f ? hi : 0.0f;
  }
  return (uint32_t)f32_to_bf16_bits(lo) | ((uint32_t)f32_to_bf16_bits(hi) << 16);
}
// Epilogue of a BF16 convolution (core/conv.cpp:90-98: fp32 result + fp32 bias, ReLU, BF16 rounding). The
// accumulators are fp32; a thread rounds two neighbouring pixels of its channel into one word, and the words are transposed
// through shared memory (see StageLane): a lane stores eight channels (16 bytes) of one pixel. `out8` addresses (pixel m0,
// this lane's group of eight channels); `ldc` is in bytes.
template <bool RELU>
__device__ __forceinline__ void epilogue_channels_bf16(const ConvGemmParams &p, uint32_t lane_addr, uint8_t *out8,
                                                       bool ch_ok, int m0, int half, int halves, unsigned long long bias2, const StageLane &st,
                                                       int ncols = 128) {
  const int cols = min(ncols, p.M_total - m0);
  int left = ch_ok ? p.M_total - m0 - half * 32 - st.px : 0; // pixels in range from this lane's first one of the chunk
  unsigned long long o = px_addr(out8, half * 32 + st.px, p.ldc);
  for (int colg = half * 32; colg < cols; colg += 32 * halves, left -= 32 * halves, o = px_addr((const void *)o, 32 * halves, p.ldc)) {
    uint32_t acc0[16], acc1[16];
    ptx::tcgen05_ld_x16(lane_addr + (uint32_t)colg, acc0);
    ptx::tcgen05_ld_x16(lane_addr + (uint32_t)colg + 16u, acc1);
    ptx::tcgen05_wait_ld();
    uint32_t w[16], odd = 0u;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      unsigned long long v = pack_b32x2(j < 8 ? acc0[2 * j] : acc1[2 * j - 16], j < 8 ? acc0[2 * j + 1] : acc1[2 * j - 15]);
      asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(bias2));
      w[j] = bf16_pack_relu<RELU>(v, odd);
    }
    if (odd & 0x7fff7fffu) {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        w[j] = bf16_pack_rule<RELU>(j < 8 ? acc0[2 * j] : acc1[2 * j - 16], j < 8 ? acc0[2 * j + 1] : acc1[2 * j - 15], __uint_as_float((uint32_t)bias2));
    }
#pragma unroll
    for (int part = 0; part < 2; ++part) { // 16 pixels each: 1 KB
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 2; ++k)
        asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(st.put + 512u * k),
                     "r"(w[8 * part + 4 * k]), "r"(w[8 * part + 4 * k + 1]), "r"(w[8 * part + 4 * k + 2]), "r"(w[8 * part + 4 * k + 3])
                     : "memory");
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        uint32_t v[4];
        lds128(st.get + 512u * k, v);
        if (16 * part + 8 * k < left)
          asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(px_addr((const void *)o, 16 * part + 8 * k, p.ldc)), "r"(v[0]),
                       "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
      }
    }
  }
}

// The same with the BF16 eltwise add (two operands, ReLU) that consumes this convolution (core/eltwise.cpp:41-52): both tensors
// are written. The sum of two BF16 values rounded once is what the reference's fp32 sum rounded to BF16 is: where the exponents
// are so far apart that the fp32 sum is inexact, the smaller operand moves neither. Residual words a chunk ahead, as in
// epilogue_add_fq. `left`: pixels in range from this lane's first one (0: the lane has no channels).
__device__ __forceinline__ void fetch_residual16(uint4 (&y)[4], const uint8_t *at, int left, int pitch) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int px = 16 * (i >> 1) + 2 * (i & 1);
    if (px < left)
      asm volatile("ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(y[i].x), "=r"(y[i].y), "=r"(y[i].z), "=r"(y[i].w) : "l"(px_addr(at, px, pitch)));
  }
}
__device__ __forceinline__ uint32_t add_relu_bf16x2(uint32_t x, uint32_t y, uint32_t &odd) {
  uint32_t s;
  asm("fma.rn.relu.bf16x2 %0, %1, %2, %3;" : "=r"(s) : "r"(x), "r"(0x3f803f80u), "r"(y));
  asm("fma.rn.bf16x2 %0, %1, %2, %0;" : "+r"(odd) : "r"(s), "r"(0u));
  return s;
}
__device__ __forceinline__ uint32_t add_relu_bf16x2_rule(uint32_t x, uint32_t y) {
  float lo = __fadd_rn(bits_f32(x << 16), bits_f32(y << 16)), hi = __fadd_rn(bits_f32(x & 0xffff0000u), bits_f32(y & 0xffff0000u));
  lo = lo > 0.0f ? lo : 0.0f;
  hi = hi > 0.0f ? hi : 0.0f;
  return (uint32_t)f32_to_bf16_bits(lo) | ((uint32_t)f32_to_bf16_bits(hi) << 16);
}
__device__ __forceinline__ void epilogue_add_bf16(const ConvGemmParams &p, uint32_t lane_addr, uint8_t *out16, int left, bool mine, int m0, int half,
                                                  unsigned long long bias2, const AddLane &al, int ncols, uint4 (&y)[4], const uint8_t *next,
                                                  int next_left) {
  const int col0 = half * 32, col1 = col0 + 64;
  const unsigned long long to_sum = (unsigned long long)(p.out2 - p.out);
  auto meet = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory"); };
  auto chunk = [&](int colg, const uint4 (&res)[4]) {
    const unsigned long long o = px_addr(out16, colg, p.ldc);
    // sixteen pixels at a time: with all 32 accumulators of the chunk beside the residual words of two, registers spilled
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      uint32_t w[8];
      if (mine) {
        uint32_t acc[16], odd = 0u;
        ptx::tcgen05_ld_x16(lane_addr + (uint32_t)(colg + 16 * part), acc);
        ptx::tcgen05_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          unsigned long long v = pack_b32x2(acc[2 * j], acc[2 * j + 1]);
          asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(bias2));
          w[j] = bf16_pack_relu<false>(v, odd);
        }
        if (odd & 0x7fff7fffu) {
#pragma unroll
          for (int j = 0; j < 8; ++j) w[j] = bf16_pack_rule<false>(acc[2 * j], acc[2 * j + 1], __uint_as_float((uint32_t)bias2));
        }
      }
      meet(); // the pixels before have been read
      if (mine) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
          asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(al.put + 512u * k), "r"(w[4 * k]),
                       "r"(w[4 * k + 1]), "r"(w[4 * k + 2]), "r"(w[4 * k + 3]) : "memory");
      }
      meet();
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        uint32_t v[4];
        lds128(al.get + 128u * k, v);
        const int px = 16 * part + 2 * k;
        if (px < left - colg) {
          const unsigned long long at = px_addr((const void *)o, px, p.ldc);
          asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
          const uint4 &x = res[2 * part + k];
          const uint32_t r[4] = {x.x, x.y, x.z, x.w};
          uint32_t s[4], far = 0u;
#pragma unroll
          for (int j = 0; j < 4; ++j) s[j] = add_relu_bf16x2(v[j], r[j], far);
          if (far & 0x7fff7fffu) {
#pragma unroll
            for (int j = 0; j < 4; ++j) s[j] = add_relu_bf16x2_rule(v[j], r[j]);
          }
          asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(at + to_sum), "r"(s[0]), "r"(s[1]), "r"(s[2]), "r"(s[3]) : "memory");
        }
      }
    }
  };
  uint4 y1[4];
  const bool two = col1 < ncols && m0 + col1 < p.M_total;
  if (two)
    fetch_residual16(y1, reinterpret_cast<const uint8_t *>(p.res) + (out16 - reinterpret_cast<uint8_t *>(p.out)) + (size_t)col1 * p.ldc,
                     left - col1, p.ldc);
  if (col0 < ncols && m0 + col0 < p.M_total) chunk(col0, y);
  fetch_residual16(y, next + (size_t)col0 * p.ldc, next_left - col0, p.ldc);
  if (two) chunk(col1, y1);
}

// Epilogue of an fp32 convolution computed as three TF32 products (calibration forward; core/conv.cpp:80-89): fp32
// accumulator + fp32 bias, ReLU, stored as fp32. A lane owns a channel: for every pixel the warp writes 32 consecutive
// channels (128 contiguous bytes). `out_ch` addresses (pixel m0, this lane's channel); `pitch` is the row pitch in bytes.
template <bool RELU>
__device__ __forceinline__ void epilogue_channels_f32(const ConvGemmParams &p, uint32_t lane_addr, uint8_t *out_ch, bool ch_ok,
                                                      int m0, int half, int halves, float bias, int ncols = 128) {
  const int cols = min(ncols, p.M_total - m0);
  int left = ch_ok ? p.M_total - m0 - half * 32 : 0; // pixels in range from the chunk's first one
  unsigned long long o = px_addr(out_ch, half * 32, p.ldc);
  const unsigned long long to_lo = (unsigned long long)(reinterpret_cast<uint8_t *>(p.out2) - reinterpret_cast<uint8_t *>(p.out));
  for (int colg = half * 32; colg < cols; colg += 32 * halves, left -= 32 * halves, o = px_addr((const void *)o, 32 * halves, p.ldc)) {
    uint32_t acc0[16], acc1[16];
    ptx::tcgen05_ld_x16(lane_addr + (uint32_t)colg, acc0);
    ptx::tcgen05_ld_x16(lane_addr + (uint32_t)colg + 16u, acc1);
    ptx::tcgen05_wait_ld();
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      float v = __fadd_rn(bits_f32(j < 16 ? acc0[j & 15] : acc1[j & 15]), bias);
      if (RELU) v = v > 0.0f ? v : 0.0f;
      if (j < left) {
        const unsigned long long at = px_addr((const void *)o, j, p.ldc);
        asm volatile("st.global.f32 [%0], %1;" ::"l"(at), "f"(v) : "memory");
        // the remainder operand of a TF32 x 3 convolution that reads this result, when one does
        if (p.out2)
          asm volatile("st.global.f32 [%0], %1;" ::"l"(at + to_lo), "f"(__fsub_rn(v, __uint_as_float(__float_as_uint(v) & 0xffffe000u))) : "memory");
      }
    }
  }
}

// Persistent kernel: gridDim.x CTAs walk the tile list (tile = blockIdx.x + k * gridDim.x; n-tiles
// vary fastest so that CTAs working at the same time share activation tiles through L2). The
// producer runs ahead through the shared-memory ring across tile boundaries and the accumulator is
// double-buffered in TMEM, so the loads and MMAs of tile i+1 overlap the epilogue of tile i.
// TF32: an fp32 convolution as three kind::tf32 products accumulated in one pass over K: with x = xh + xl and
// w = wh + wl (h: the upper 19 bits of the fp32 word, l: the exact remainder), x w = xh wh + xl wh + xh wl up to
// 2^-22 relative. The K loop runs three times over the taps: term 0 reads (tmA2, tmB) = (xl, wh), term 1
// (tmA, tmB2) = (xh, wl), term 2 (tmA, tmB) = (xh, wh); the accumulator never leaves TMEM in between. The two small
// terms come first: the tensor core truncates every partial sum at the accumulator's own precision, so each MMA
// step costs up to an ulp of what has been accumulated so far, and only the steps of the last term see the
// full magnitude (measured: the error against a double-accumulated convolution drops by the expected factor 3).
template <bool BF16, bool FAST = true, bool TF32 = false, bool SPLIT = false, int ACTSEL = -1>
__device__ __forceinline__ void conv_gemm_body(const CUtensorMap &tmA, const CUtensorMap &tmB, const ConvGemmParams &p,
                                               const CUtensorMap &tmA2, const CUtensorMap &tmB2) {
  constexpr int KIND = TF32 ? 2 : (BF16 ? 1 : 0);
  constexpr int kTerms = TF32 ? 3 : 1;
  constexpr bool FQ = ACTSEL >= 100; // one epilogue, the floating-point requantisation: ACTSEL - 100 is the activation
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (base - raw);

  // header layout
  const uint32_t bar_full = base;             // kMaxStages x 8 B
  const uint32_t bar_empty = base + 64;       // kMaxStages x 8 B
  const uint32_t bar_acc_full = base + 128;   // 2 x 8 B: accumulator buffer complete
  const uint32_t bar_acc_empty = base + 144;  // 2 x 8 B: accumulator buffer drained by the epilogue
  const uint32_t bar_w = base + 160;          // resident weights landed
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 168);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 172);
  volatile int *split_last = reinterpret_cast<volatile int *>(smem + 176); // split K: this CTA completes its tile

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const int n_tiles = (p.n_valid + p.BN - 1) / p.BN;
  // Dual mode (<= 64 output channels): a tile covers 256 pixels. The weight tile is fetched as 192 rows
  // starting 64 rows BEFORE the first channel, i.e. [64 zero rows][64 weight rows][64 zero rows]; rows
  // 64..191 of it ([W; 0]) times the first 128 pixels fill TMEM lanes 0..63, rows 0..127 ([0; W]) times
  // the second 128 pixels accumulate into lanes 64..127, so all 128 lanes (and all epilogue warps) work.
  const int m_tile = p.m_tile, ncols = p.dual ? 128 : m_tile;
  const int m_tiles = (p.M_total + m_tile - 1) / m_tile;
  int total_tiles = n_tiles * m_tiles; // set to 0 below when the launch is already marked as failed
  const uint32_t a_bytes = (uint32_t)m_tile * (uint32_t)p.BK;
  const uint32_t b_bytes = (uint32_t)(p.dual ? 192 : p.BN) * (uint32_t)p.BK;
  const int taps = p.kh * p.kw;
  const int k_iters = taps * p.c_chunks;
  // Weight-resident mode: [all K blocks of the weights][ring of activation tiles]; the launch grid is a
  // multiple of the channel-tile count, so a CTA's channel tile never changes. Otherwise the ring
  // holds (activation tile, weight tile) pairs.
  const uint32_t w_base = base + kSmemHeader;
  const uint32_t tiles = p.w_resident ? w_base + (uint32_t)k_iters * b_bytes : w_base;
  const uint32_t stage_bytes = p.w_resident ? a_bytes : a_bytes + b_bytes;
  const uint32_t acc_stride = (uint32_t)(p.tmem_cols >> 1); // columns per accumulator buffer
  // The tile walk (tile = blockIdx.x + k * gridDim.x, channel tiles fastest) as a running (pixel tile, channel tile)
  // pair: the per-tile code of every role carries no division.
  const int walk_m0 = (int)blockIdx.x / n_tiles, walk_n0 = (int)blockIdx.x % n_tiles;
  const int walk_dm = (int)gridDim.x / n_tiles, walk_dn = (int)gridDim.x % n_tiles;
  const int wait_rounds = p.wait_rounds > 0 ? p.wait_rounds : 1024;
  // split K: a work item is (tile, K range); item = tile * split_k + range, one loop over items in every role
  const int split_k = (!SPLIT || p.split_k < 1) ? 1 : p.split_k; // SPLIT is a compile-time switch: the ordinary kernels carry none of it

  // Programmatic dependent launch: the next kernel of the stream may start its own set-up as soon as every CTA
  // of this launch has got here; this kernel in turn sets up its barriers and tensor memory while the
  // previous one is still finishing and only then waits for that kernel's results (pdl_wait below).
  pdl_trigger();
  if (threadIdx.x == 0) {
    // A CTA of a launch in which an earlier CTA already gave up does no work at all, so that a broken launch ends
    // quickly instead of timing out once per tile. The flag is read first and stored last, so that the load's
    // latency passes behind the barrier set-up, and ahead of pdl_wait on purpose: a flag raised by the previous
    // kernel after this read only costs this CTA its own bounded wait, the host sees the error either way.
    const int gave_up = *reinterpret_cast<volatile int *>(p.err);
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(bar_full + 8 * s, 1);
      ptx::mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(bar_acc_full + 8 * b, 1);
      ptx::mbar_init(bar_acc_empty + 8 * b, kEpilogueWarps);
    }
    ptx::mbar_init(bar_w, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *abort_flag = gave_up;
  }
  if (warp == 1) {
    ptx::tcgen05_alloc(ptx::smem_u32(tmem_slot), (uint32_t)p.tmem_cols);
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  if (*abort_flag != 0) total_tiles = 0;
  const int total_items = total_tiles * split_k;
  // What does not depend on the previous kernel is started before the wait for it: the tensor maps are fetched and a
  // CTA that keeps its weights resident starts their copies (weights are written at load time only).
  if (warp == 0 && ptx::elect_one()) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB) : "memory");
    if (p.w_resident && (int)blockIdx.x < total_tiles) {
      const int n0w = ((int)blockIdx.x % n_tiles) * p.BN - (p.dual ? 64 : 0);
      ptx::mbar_expect_tx(bar_w, (uint32_t)k_iters * b_bytes);
      for (int kit = 0; kit < k_iters; ++kit)
        ptx::tma_load_3d(w_base + (uint32_t)kit * b_bytes, &tmB, bar_w, (kit % p.c_chunks) * p.BK, kit / p.c_chunks,
                         n0w);
    }
  }
  // From here on the kernel touches the activations: the previous kernel's writes must be complete and visible.
  pdl_wait();

  if (warp == 0) {
    // ---------------------------------------------------------------- producer
    {
      int it = 0; // k-iterations issued so far, across tiles
      int ps = 0;        // ring stage of iteration `it`
      uint32_t pph = 0;  // its phase bit
      bool ok = true;
      int tm = walk_m0, tn = walk_n0; // (resident weights: their copies were started before the wait above)
      for (int item = blockIdx.x; item < total_items && ok; item += gridDim.x) {
        int k_begin = 0, k_end = kTerms * k_iters;
        if (split_k > 1) { // few items per CTA: the divisions do not matter here
          const int tile = item / split_k;
          tm = tile / n_tiles;
          tn = tile - tm * n_tiles;
          k_begin = (item - tile * split_k) * p.k_per;
          k_end = min(k_iters, k_begin + p.k_per);
        }
        const int m0 = tm * m_tile;
        const int n0 = tn * p.BN - (p.dual ? 64 : 0);
        tm += walk_dm;
        tn += walk_dn;
        if (tn >= n_tiles) {
          tn -= n_tiles;
          ++tm;
        }
        int n_img = 0, h_base = 0, w_base = 0; // im2col: base coordinates of the tile's first pixel
        if (p.a_mode == 1) {
          const int q = m0 % p.OW;
          const int t = m0 / p.OW;
          const int pp = t % p.OH;
          n_img = t / p.OH;
          w_base = q * p.sw - p.pl;
          h_base = pp * p.sh - p.pt;
        }
        // running (tap row, tap column, channel chunk) and ring (stage, phase) counters: this loop
        // is a single thread's instruction stream, so it carries no divisions
        int tap = 0, tr = 0, ts = 0, chunk = 0, term = 0;
        if (k_begin > 0) {
          tap = k_begin / p.c_chunks;
          chunk = k_begin - tap * p.c_chunks;
          tr = tap / p.kw;
          ts = tap - tr * p.kw;
        }
        for (int kit = k_begin; kit < k_end; ++kit, ++it) {
          const CUtensorMap *mapA = (TF32 && term == 0) ? &tmA2 : &tmA;
          const CUtensorMap *mapB = (TF32 && term == 1) ? &tmB2 : &tmB;
          if (it >= p.stages && !ptx::mbar_wait_warp(bar_empty + 8 * ps, pph ^ 1u, abort_flag, wait_rounds)) {
            wait_expired(p.err, abort_flag, kErrEmptyWait);
            ok = false;
            break;
          }
          const int c0 = chunk * p.BK;
          const uint32_t a_dst = tiles + (uint32_t)ps * stage_bytes;
          const uint32_t b_dst = a_dst + a_bytes;
          const uint32_t fb = bar_full + 8 * ps;
          if (ptx::elect_one()) {
            ptx::mbar_expect_tx(fb, stage_bytes);
            if (p.a_mode == 1) {
              // one copy per tile, also in dual mode (the map's pixel count per copy is the tile's)
              ptx::tma_load_im2col_4d(a_dst, mapA, fb, c0, w_base, h_base, n_img, (uint16_t)(ts * p.dw),
                                      (uint16_t)(tr * p.dh));
            } else {
              ptx::tma_load_2d(a_dst, mapA, fb, c0, m0);
            }
            if (!p.w_resident) ptx::tma_load_3d(b_dst, mapB, fb, c0, tap, n0);
          }
          if (++chunk == p.c_chunks) {
            chunk = 0;
            ++tap;
            if (++ts == p.kw) {
              ts = 0;
              ++tr;
            }
            if (TF32 && tap == taps) { // next term: the same taps over the other operand pair
              tap = 0;
              tr = 0;
              ts = 0;
              ++term;
            }
          }
          if (++ps == p.stages) {
            ps = 0;
            pph ^= 1u;
          }
        }
      }
      if (!ok || *abort_flag) {
        if (p.w_resident && (int)blockIdx.x < total_tiles)
          for (uint32_t w = 0; w < (1u << 20); ++w)
            if (ptx::mbar_try_wait(bar_w, 0u)) break;
        // Drain: wait (bounded) until every copy this thread issued has landed, so that no bulk
        // copy is in flight when the CTA's shared memory is released.
        int first = it > p.stages ? it - p.stages : 0;
        for (int j = first; j < it; ++j) {
          const int s = j % p.stages;
          const uint32_t ph = (uint32_t)(j / p.stages) & 1u;
          for (uint32_t w = 0; w < (1u << 20); ++w)
            if (ptx::mbar_try_wait(bar_full + 8 * s, ph)) break;
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    {
      int it = 0, t = 0;
      int ms = 0;        // ring stage of iteration `it`
      uint32_t mph = 0;  // its phase bit
      bool ok = true;
      // Shared-memory descriptors differ between stages and K steps only in the start-address field of
      // their low word (16-byte units, no carry out of its 14 bits below 256 KB): the low words are
      // advanced by 32-bit adds and the issue loop stays short. A single thread feeds the tensor core,
      // and every instruction it spends per K block beyond the MMAs themselves shows up as idle tensor
      // cycles (measured: ~35 extra instructions per 4 MMAs cost a third of the MMA rate).
      const uint64_t desc_ring0 = make_kmajor_desc(tiles, p.BK);
      const uint32_t desc_hi = (uint32_t)(desc_ring0 >> 32);
      const uint32_t desc_ring_lo = (uint32_t)desc_ring0;
      const uint32_t desc_w_lo = (uint32_t)make_kmajor_desc(w_base, p.BK);
      const uint32_t stage_step = stage_bytes >> 4, a_step = a_bytes >> 4, w_step = b_bytes >> 4;
      const uint32_t sub_step = (128u * (uint32_t)p.BK) >> 4, dual_step = (64u * (uint32_t)p.BK) >> 4;
      uint32_t m_full = bar_full, m_empty = bar_empty, ring_lo = desc_ring_lo;
      const int ksteps = p.ksteps;
      if (p.w_resident && (int)blockIdx.x < total_tiles) {
        if (!ptx::mbar_wait_warp(bar_w, 0u, abort_flag, wait_rounds)) {
          wait_expired(p.err, abort_flag, kErrFullWait);
          ok = false;
        }
      }
      for (int item = blockIdx.x; item < total_items && ok; item += gridDim.x, ++t) {
        int k_begin = 0, k_end = kTerms * k_iters;
        if (split_k > 1) {
          k_begin = (item % split_k) * p.k_per;
          k_end = min(k_iters, k_begin + p.k_per);
        }
        const int buf = t & 1;
        if (t >= 2) {
          // the epilogue must have drained this accumulator buffer (its previous use)
          if (!ptx::mbar_wait_warp(bar_acc_empty + 8 * buf, (uint32_t)(((t >> 1) - 1) & 1), abort_flag, wait_rounds)) {
            wait_expired(p.err, abort_flag, kErrAccWait);
            ok = false;
            break;
          }
          ptx::tcgen05_fence_after();
        }
        const uint32_t d_tmem = tmem_base + (uint32_t)buf * acc_stride;
        uint32_t wres_lo = desc_w_lo; // weight-resident mode: descriptor (low word) of K block `kit`
        // The loop over K blocks twice: for whole blocks of plain tiles, and for blocks with a padded tail and dual mode. One
        // loop that chose between one and four MMAs inside cost every K block 23 ns (3x3, 512 channels, 7x7, N = 1 unsplit,
        // 36 blocks: 15.4 -> 13.9 us; ResNet-50 batch 1 318 -> 292 us, batch 256 2560 -> 2530).
        auto k_loop = [&](auto whole) {
          for (int kit = k_begin; kit < k_end; ++kit, ++it) {
            if (!ptx::mbar_wait_warp(m_full, mph, abort_flag, wait_rounds)) {
              wait_expired(p.err, abort_flag, kErrFullWait);
              ok = false;
              break;
            }
            ptx::tcgen05_fence_after();
            // transposed product: weights are the A operand (M = channels), activations B (N = pixels)
            const uint32_t w_lo = p.w_resident ? wres_lo : ring_lo + a_step;
            const uint32_t acc_first = kit > k_begin ? 1u : 0u;
            if (ptx::elect_one()) {
              if constexpr (decltype(whole)::value) {
                ptx::tcgen05_mma_i8_kblock<4, KIND>(d_tmem, w_lo, ring_lo, desc_hi, p.idesc, acc_first);
              } else if (!p.dual) {
                if (ksteps == 3) ptx::tcgen05_mma_i8_kblock<3, KIND>(d_tmem, w_lo, ring_lo, desc_hi, p.idesc, acc_first);
                else if (ksteps == 2) ptx::tcgen05_mma_i8_kblock<2, KIND>(d_tmem, w_lo, ring_lo, desc_hi, p.idesc, acc_first);
                else ptx::tcgen05_mma_i8_kblock<1, KIND>(d_tmem, w_lo, ring_lo, desc_hi, p.idesc, acc_first);
              } else {
                // dual mode: sub-tile 0 uses weight rows 64..191 ([W; 0]), sub-tile 1 rows 0..127 ([0; W])
                for (int sub = 0; sub < 2; ++sub) {
                  const uint32_t a_lo = w_lo + (sub == 0 ? dual_step : 0u);
                  const uint32_t b_lo = ring_lo + (uint32_t)sub * sub_step;
                  const uint32_t first = (kit > k_begin || sub > 0) ? 1u : 0u;
                  if (ksteps == 4) ptx::tcgen05_mma_i8_kblock<4, KIND>(d_tmem, a_lo, b_lo, desc_hi, p.idesc, first);
                  else if (ksteps == 3) ptx::tcgen05_mma_i8_kblock<3, KIND>(d_tmem, a_lo, b_lo, desc_hi, p.idesc, first);
                  else if (ksteps == 2) ptx::tcgen05_mma_i8_kblock<2, KIND>(d_tmem, a_lo, b_lo, desc_hi, p.idesc, first);
                  else ptx::tcgen05_mma_i8_kblock<1, KIND>(d_tmem, a_lo, b_lo, desc_hi, p.idesc, first);
                }
              }
              ptx::tcgen05_commit(m_empty); // frees the stage when the MMAs retire
            }
            wres_lo += w_step;
            m_full += 8;
            m_empty += 8;
            ring_lo += stage_step;
            if (++ms == p.stages) {
              ms = 0;
              mph ^= 1u;
              m_full = bar_full;
              m_empty = bar_empty;
              ring_lo = desc_ring_lo;
            }
          }
        };
        if (ksteps == 4 && !p.dual) k_loop(std::true_type{});
        else k_loop(std::false_type{});
        if (ok && ptx::elect_one()) ptx::tcgen05_commit(bar_acc_full + 8 * buf);
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int quarter = warp & 3;     // TMEM lanes (= channels of the tile) this warp may read
    const int half = (warp - 2) >> 2; // which alternate 32-pixel column groups it takes
    const StageLane st = make_stage_lane<BF16 ? 2 : 4>(base + 1024u + (uint32_t)((warp - 2) * kStageBytes), lane);
    ChanConst cc = {};
    FloatRequantPairs<ACTSEL == 101> fq = {};
    FloatRequantShared fshared = {};
    if constexpr (FQ && ACTSEL != 101) fshared.set();
    float bias_f = 0.0f;
    unsigned long long bias2 = 0;
    int staged_n0 = -1;
    int t = 0;
    bool ok = true;
    int tm = walk_m0, tn = walk_n0;
    // fused add (INT8): this lane's first pixel of tile (m, n) in the residual, and the pixels in range from there
    uint4 res_words[2];
    const AddLane al = BF16 ? make_add_lane16(base + 256u, half, quarter, lane) : make_add_lane(base + 256u, half, quarter, lane);
    auto residual_at = [&](int m, int n) { return p.res + ((size_t)m * m_tile + al.px) * p.ldc + p.c_off + n * p.BN + al.ch; };
    auto residual_left = [&](int item, int m, int n) {
      return item < total_items && n * p.BN + al.ch < p.n_valid ? p.M_total - m * m_tile - al.px : 0;
    };
    bool live = true; // INT8 add: false once a wait has run out; the warp then does no work but comes to every barrier
    uint4 res16[4]; // the same for the BF16 add
    auto res16_at = [&](int m, int n) {
      return reinterpret_cast<const uint8_t *>(p.res) + ((size_t)m * m_tile + al.px) * p.ldc + (size_t)(n * p.BN + al.ch) * 2;
    };
    constexpr bool ADD = ACTSEL == 103 || (BF16 && ACTSEL == 3);
    if constexpr (BF16 && ACTSEL == 3)
      fetch_residual16(res16, res16_at(tm, tn) + (size_t)(half * 32) * p.ldc, residual_left(blockIdx.x, tm, tn) - half * 32, p.ldc);
    if constexpr (ACTSEL == 103) {
      fetch_residual(res_words, residual_at(tm, tn) + (size_t)(half * 32) * p.ldc, residual_left(blockIdx.x, tm, tn) - half * 32, p.ldc);
    }
    for (int item = blockIdx.x; item < total_items && ok; item += gridDim.x, ++t) {
      int tile = item;
      if (split_k > 1) {
        tile = item / split_k;
        tm = tile / n_tiles;
        tn = tile - tm * n_tiles;
      }
      // dual mode: lanes 0..63 are the channels of the first 128 pixels, lanes 64..127 of the second
      // pixel groups: lane / (128 / group) is the pixel of the group
      const int ch_base = p.dual ? (quarter & 1) * 32 : (p.group > 1 ? (quarter * 32) & (128 / p.group - 1) : quarter * 32);
      const int m0 = tm * m_tile + (p.dual ? 128 * (quarter >> 1) : 0);
      const int n0 = tn * p.BN;
      tm += walk_dm;
      tn += walk_dn;
      if (tn >= n_tiles) {
        tn -= n_tiles;
        ++tm;
      }
      const int buf = t & 1;
      if (n0 != staged_n0) {
        if (BF16 || TF32) {
          const int ch = n0 + ch_base + lane_channel(lane);
          bias_f = ch < p.n_valid ? __int_as_float(p.bias[ch]) : 0.0f; // fp32 bias bits in the int32 array
          if (BF16) bias2 = hold_pair(bias_f);
        } else if (FQ) {
          const int ch = n0 + ch_base + lane_channel(lane);
          const uint4 c = ch < p.n_valid ? __ldg(reinterpret_cast<const uint4 *>(p.fq) + ch) : make_uint4(0u, 0u, 0u, 0u);
          fq.set(FloatRequant{c.x, __uint_as_float(c.y), __uint_as_float(c.z), __uint_as_float(c.w)});
        } else {
          cc = load_chan_const(p, n0 + ch_base + lane_channel(lane));
        }
        staged_n0 = n0;
      }
      ok = live && ptx::mbar_wait_bounded(bar_acc_full + 8 * buf, (uint32_t)((t >> 1) & 1), abort_flag, wait_rounds);
      if (!ok && !*abort_flag) {
        report_error(p.err, kErrAccWait);
        *abort_flag = 1;
      }
      // the wait result may differ between lanes only on the error path; make it uniform
      ok = __all_sync(0xffffffffu, ok);
      if constexpr (ADD) {
        live = ok;
        ok = true;
      }
      const bool split_item = SPLIT && split_k > 1;
      if (!ok && !split_item) break; // (a split item still passes its two barriers, see below)
      ptx::tcgen05_fence_after();
      const int ch8 = n0 + ch_base + (lane & 3) * 8;
      int32_t *ws_lane = nullptr; // split K: this lane's channel column of the tile's partial-sum block
      if (split_item) {
        ws_lane = p.ws + (size_t)tile * (128 * 128) + quarter * 32 + lane;
        if (ok && n0 + ch_base < p.n_valid && m0 < p.M_total) {
          // this CTA's partial accumulator goes to the tile's block in global memory (one reduction per value,
          // 128 contiguous bytes per warp and column)
          const uint32_t lane_addr = tmem_base + (uint32_t)buf * acc_stride + ((uint32_t)(quarter * 32) << 16);
          for (int colg = half * 32; colg < ncols; colg += 32 * (kEpilogueWarps / 4)) {
            if (m0 + colg >= p.M_total) break;
            uint32_t a0[16], a1[16];
            ptx::tcgen05_ld_x16(lane_addr + (uint32_t)colg, a0);
            ptx::tcgen05_ld_x16(lane_addr + (uint32_t)colg + 16u, a1);
            ptx::tcgen05_wait_ld();
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              atomicAdd(ws_lane + (size_t)(colg + k) * 128, (int)a0[k]);
              atomicAdd(ws_lane + (size_t)(colg + 16 + k) * 128, (int)a1[k]);
            }
          }
        }
        // the accumulator buffer is free again
        ptx::tcgen05_fence_before();
        __syncwarp();
        if (ok && lane == 0 && !p.lose_arrival)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_acc_empty + 8 * buf) : "memory");
        // Count this CTA in once all of its epilogue warps have added their part; the CTA that completes the tile
        // goes on to the epilogue proper, the others are done with it (nobody waits for another CTA). The two
        // barriers are among the epilogue warps of this CTA only, and every one of them reaches both: a warp whose
        // wait ran out has raised the abort flag before the first, the leader turns that into "stop" for all (2),
        // so that no warp goes on to a barrier the others will not come to.
        __threadfence();
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpilogueWarps) : "memory");
        if (warp == 2 && lane == 0) {
          int verdict = 2;
          if (!*abort_flag) {
            const unsigned int before = atomicAdd(p.ws_count + tile, 1u);
            verdict = before == (unsigned int)(split_k - 1) ? 1 : 0;
            if (verdict) p.ws_count[tile] = 0u; // ready for the next launch
          }
          *split_last = verdict;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpilogueWarps) : "memory");
        const int verdict = *split_last;
        if (verdict == 2) {
          ok = false;
          break;
        }
        if (verdict == 0) continue;
        __threadfence();
      }
      if ((ADD || n0 + ch_base < p.n_valid) && m0 < p.M_total) { // warp-uniform: this lane quarter holds real outputs
        const uint32_t lane_addr = tmem_base + (uint32_t)buf * acc_stride + ((uint32_t)(quarter * 32) << 16);
        const size_t out_m0 = (size_t)m0 * p.ldc + (p.group > 1 ? (quarter * 32 * p.group >> 7) * p.ldc_px : 0); // bytes
        int8_t *out8 = p.out + out_m0 + p.c_off + ch8;
        const bool ch8_ok = ch8 < p.n_valid;
        if (TF32) {
          // byte addressing: 4 bytes per channel
          const int ch = n0 + ch_base + lane_channel(lane);
          uint8_t *out_ch = reinterpret_cast<uint8_t *>(p.out) + out_m0 + (size_t)(p.c_off + ch) * 4;
          if (p.act == 1) epilogue_channels_f32<true>(p, lane_addr, out_ch, ch < p.n_valid, m0, half, kEpilogueWarps / 4, bias_f, ncols);
          else epilogue_channels_f32<false>(p, lane_addr, out_ch, ch < p.n_valid, m0, half, kEpilogueWarps / 4, bias_f, ncols);
        } else if (BF16) {
          // byte addressing: 2 bytes per channel
          uint8_t *out16 = reinterpret_cast<uint8_t *>(p.out) + out_m0 + (size_t)(p.c_off + ch8) * 2;
          if constexpr (ACTSEL == 3)
            epilogue_add_bf16(p, lane_addr, reinterpret_cast<uint8_t *>(p.out) + (size_t)(m0 + al.px) * p.ldc + (size_t)(n0 + al.ch) * 2,
                              live && n0 + al.ch < p.n_valid ? p.M_total - m0 - al.px : 0, live && n0 + ch_base < p.n_valid, m0, half, bias2,
                              al, ncols, res16, res16_at(tm, tn), residual_left(item + gridDim.x, tm, tn));
          else if (p.act == 1) epilogue_channels_bf16<true>(p, lane_addr, out16, ch8_ok, m0, half, kEpilogueWarps / 4, bias2, st, ncols);
          else epilogue_channels_bf16<false>(p, lane_addr, out16, ch8_ok, m0, half, kEpilogueWarps / 4, bias2, st, ncols);
        } else if constexpr (ACTSEL == 103) {
          epilogue_add_fq(p, lane_addr, p.out + (size_t)(m0 + al.px) * p.ldc + p.c_off + n0 + al.ch,
                          live && n0 + al.ch < p.n_valid ? p.M_total - m0 - al.px : 0, live && n0 + ch_base < p.n_valid, m0, half, fq, fshared, al,
                          ncols, res_words, residual_at(tm, tn), residual_left(item + gridDim.x, tm, tn));
        } else if constexpr (FQ) {
          epilogue_channels_impl<ACTSEL - 100, 3>(p, lane_addr, out8, ch8_ok, m0, half, kEpilogueWarps / 4, lane, fq, fshared, st, ncols);
        } else if (p.act == 1) epilogue_channels_impl<1, FAST ? 1 : 0, SPLIT>(p, lane_addr, out8, ch8_ok, m0, half, kEpilogueWarps / 4, lane, cc, fshared, st, ncols, ws_lane);
        else if (p.act == 2) epilogue_channels_impl<2, FAST ? 1 : 0, SPLIT>(p, lane_addr, out8, ch8_ok, m0, half, kEpilogueWarps / 4, lane, cc, fshared, st, ncols, ws_lane);
        else if (p.act == 3) epilogue_channels_impl<3, FAST ? 1 : 0>(p, lane_addr, out8, ch8_ok, m0, half, kEpilogueWarps / 4, lane, cc, fshared, st, ncols);
        else if (FAST && (p.fastq & 2)) epilogue_channels_impl<0, FAST ? 2 : 0, SPLIT>(p, lane_addr, out8, ch8_ok, m0, half, kEpilogueWarps / 4, lane, cc, fshared, st, ncols, ws_lane);
        else epilogue_channels_impl<0, FAST ? 1 : 0, SPLIT>(p, lane_addr, out8, ch8_ok, m0, half, kEpilogueWarps / 4, lane, cc, fshared, st, ncols, ws_lane);
      }
      if (SPLIT && ws_lane) continue; // split K: the accumulator buffer was handed back above
      // hand the accumulator buffer back to the MMA issuer
      ptx::tcgen05_fence_before();
      __syncwarp();
      if (lane == 0 && !p.lose_arrival)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_acc_empty + 8 * buf) : "memory");
    }
  }

  ptx::tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tcgen05_fence_after();
    ptx::tcgen05_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
}

// p.fastq bit 0 must be set: the epilogue uses the multiply-high requantisation (requant_fast)
__global__ void __launch_bounds__(kConvThreads, 2)
conv_gemm_i8_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const ConvGemmParams p) {
  conv_gemm_body<false, true>(tmA, tmB, p, tmA, tmB);
}
// The floating-point requantisation (p.fq set), one kernel per activation (ConvGemmParams::act): the compiler allocates
// registers and schedules for that one epilogue.
template <int ACT>
__global__ void __launch_bounds__(kConvThreads, 2)
conv_gemm_i8_fq_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                       const ConvGemmParams p) {
  conv_gemm_body<false, true, false, false, 100 + ACT>(tmA, tmB, p, tmA, tmB);
}
// The split-K form of both (ConvGemmParams::split_k > 1): a kernel of its own, so that the ordinary ones carry none of
// its code (with the switch at run time the epilogue-bound layers were 14% slower).
template <bool FAST>
__global__ void __launch_bounds__(kConvThreads, 2)
conv_gemm_i8_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          const ConvGemmParams p) {
  conv_gemm_body<false, FAST, false, true>(tmA, tmB, p, tmA, tmB);
}
// the same with the 64-bit multiply-add requantisation (requant_one), for layers outside requant_fast's domain
__global__ void __launch_bounds__(kConvThreads, 2)
conv_gemm_i8_wide_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                         const ConvGemmParams p) {
  conv_gemm_body<false, false>(tmA, tmB, p, tmA, tmB);
}
// The same pipeline for BF16 graphs: BF16 operands (tcgen05 kind::f16), fp32 accumulators, BF16 results.
// All sizes in ConvGemmParams that count K or row pitches are in BYTES, so only the MMA kind and the
// epilogue differ.
__global__ void __launch_bounds__(kConvThreads, 2)
conv_gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const ConvGemmParams p) {
  conv_gemm_body<true, false>(tmA, tmB, p, tmA, tmB);
}
// ... with the residual add that consumes it (ConvGemmParams::act 3)
__global__ void __launch_bounds__(kConvThreads, 2)
conv_gemm_bf16_add_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          const ConvGemmParams p) {
  conv_gemm_body<true, false, false, false, 3>(tmA, tmB, p, tmA, tmB);
}

// fp32 convolution on the tensor cores as three TF32 products (see conv_gemm_body): tmA / tmA2 are the upper and
// the remainder part of the activations, tmB / tmB2 of the weights.
__global__ void __launch_bounds__(kConvThreads, 2)
conv_gemm_tf32x3_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                        const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB2,
                        const ConvGemmParams p) {
  conv_gemm_body<false, false, true>(tmA, tmB, p, tmA2, tmB2);
}

// x -> remainder x - (upper 19 bits of x), exact; the upper part is what a kind::tf32 product reads of x itself.
__global__ void tf32_split_kernel(const float4 *__restrict__ x, float4 *__restrict__ lo, size_t nvec) {
  pdl_prologue();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nvec; i += (size_t)gridDim.x * blockDim.x) lo[i] = tf32_remainder(x[i]);
}

} // namespace tpucb
