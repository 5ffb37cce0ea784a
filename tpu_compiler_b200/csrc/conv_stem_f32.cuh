// The image stem of an fp32 network (at most 4 input channels, at most 64 outputs) on the tensor cores, as three TF32 products
// (see conv_gemm_body), from patches that are built in shared memory.
//
// A tap of a pixel is one 16-byte vector of the NHWC4 image. Written to memory as a patch matrix, with its remainder part beside
// it, the patches of ResNet-50's stem are 2 x 630 MB for 64 images, which the product then read three times: 877 us, nearly all
// of it memory traffic. Here eight warps fetch the taps of 64 pixels (through L1, where neighbouring pixels find them again),
// form the remainders and store both in the layout of unswizzled operands: per tap 64 rows of 16 bytes, so that a step of
// kind::tf32 (32 bytes of K) takes two taps. The weights, high and remainder parts, stay in shared memory. The order of the
// sums is that of the patch matrix: terms, then taps, then channels, 8 values per step. The tensor core then bounds it: 75 steps
// per 64 pixels, half of their 128 rows past the 64 channels.
//
// Warps (448 threads): 0..7 build patches, 8, 9, 12, 13 are the epilogue (two quarters of 32 channels x two groups of 32
// pixels), 10 owns tensor memory and issues the MMAs. The remainder tile of the next pixels is filled while the two products
// with the high part run, the high part's while the next remainder product does.
#pragma once
#include "conv_gemm_i8.cuh"

namespace tpucb {

constexpr int kStemThreads = 448;
constexpr int kStemPx = 64;
constexpr int kStemMaxTaps = 54;                            // four operands of 1 KB per tap: 216 KB
constexpr int kStemPasses = (kStemMaxTaps + 3) / 4;         // 256 threads: 64 pixels x 4 taps at a time
constexpr int kStemHeader = 1024;                           // barriers, then the taps' offsets

struct StemArgs {
  const float4 *in;
  const uint8_t *w; // [2][taps, even][64 channels][4 floats]: high parts, remainders
  int ih, iw, taps; // p.kh x p.kw
};
inline size_t stem_smem(int taps) { return 1024 + kStemHeader + (size_t)(taps + 1) / 2 * 2 * 1024 * 4 + 1024; }

template <bool RELU>
__global__ void __launch_bounds__(kStemThreads, 1) conv_stem_tf32x3_kernel(const StemArgs a, const ConvGemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (base - raw);
  const uint32_t bar_full = base, bar_empty = base + 16; // [0] remainders, [1] high parts
  const uint32_t bar_acc_full = base + 32, bar_acc_empty = base + 48, bar_w = base + 64;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 72);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 76);
  int *tab = reinterpret_cast<int *>(smem + 128); // per tap: row and column offset, 16 bits each
  const int taps2 = (a.taps + 1) / 2 * 2;
  const uint32_t part = (uint32_t)taps2 * 1024u;
  const uint32_t wgt = base + kStemHeader, act = wgt + 2 * part; // wh, wl; xl, xh

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  int tiles = (p.M_total + kStemPx - 1) / kStemPx;
  const int wait_rounds = p.wait_rounds > 0 ? p.wait_rounds : 1024;
  pdl_trigger();
  if (threadIdx.x == 0) {
    const int gave_up = *reinterpret_cast<volatile int *>(p.err); // as in conv_gemm_body
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(bar_full + 8 * i, 8);
      ptx::mbar_init(bar_empty + 8 * i, 1);
      ptx::mbar_init(bar_acc_full + 8 * i, 1);
      ptx::mbar_init(bar_acc_empty + 8 * i, 4);
    }
    ptx::mbar_init(bar_w, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *abort_flag = gave_up;
    ptx::mbar_expect_tx(bar_w, 2 * part); // written at load time only: the copy need not wait for the previous kernel
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(wgt), "l"(a.w),
                 "r"(2 * part), "r"(bar_w) : "memory");
  }
  if (threadIdx.x < a.taps) tab[threadIdx.x] = (threadIdx.x / p.kw) * p.dh << 16 | (threadIdx.x % p.kw) * p.dw;
  if (a.taps != taps2 && threadIdx.x < 2 * kStemPx) // the tap that only fills the last step: zeros
    *reinterpret_cast<float4 *>(smem + kStemHeader + (2 + threadIdx.x / kStemPx) * part + (size_t)a.taps * 1024 + threadIdx.x % kStemPx * 16) =
        make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 10) ptx::tcgen05_alloc(ptx::smem_u32(tmem_slot), 128u);
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  if (*abort_flag != 0) tiles = 0;

  if (warp < 8) {
    // ------------------------------------------------------------------------------------------------------- patches
    const int px = threadIdx.x & (kStemPx - 1), tap0 = threadIdx.x >> 6;
    pdl_wait();
    int t = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++t) {
      const int m = tile * kStemPx + px;
      int x0 = 0, y0 = 1 << 28; // past the last pixel: every tap outside the image
      const float4 *img = a.in;
      if (m < p.M_total) {
        const int q = m % p.OW, r = m / p.OW, y = r % p.OH;
        img += (size_t)(r / p.OH) * a.ih * a.iw;
        x0 = q * p.sw - p.pl;
        y0 = y * p.sh - p.pt;
      }
      float4 v[kStemPasses];
#pragma unroll
      for (int i = 0; i < kStemPasses; ++i) {
        const int tap = tap0 + 4 * i;
        v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (tap < a.taps) {
          const int o = tab[tap], y = y0 + (o >> 16), x = x0 + (o & 0xffff);
          if ((unsigned)y < (unsigned)a.ih && (unsigned)x < (unsigned)a.iw) v[i] = __ldg(img + (size_t)y * a.iw + x);
        }
      }
      bool ok = true;
#pragma unroll
      for (int h = 0; h < 2; ++h) { // the remainders, then the high parts: the tensor core reads the upper 19 bits of the value itself
        if (t > 0 && !ptx::mbar_wait_warp(bar_empty + 8 * h, (uint32_t)((t - 1) & 1), abort_flag, wait_rounds)) {
          wait_expired(p.err, abort_flag, kErrEmptyWait);
          ok = false;
          break;
        }
        const uint32_t to = act + h * part + (uint32_t)px * 16u;
#pragma unroll
        for (int i = 0; i < kStemPasses; ++i) {
          const int tap = tap0 + 4 * i;
          if (tap < a.taps) {
            const float4 w = h ? v[i] : tf32_remainder(v[i]);
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + (uint32_t)tap * 1024u), "f"(w.x), "f"(w.y), "f"(w.z), "f"(w.w)
                         : "memory");
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_full + 8 * h) : "memory");
      }
      if (!ok) break;
    }
  } else if (warp == 10) {
    // ---------------------------------------------------------------------------------------------------- MMA issuer
    // unswizzled operand: 8 rows x 16 bytes lie together, the next 8 rows 128 bytes on, the next 16 bytes of K 1024
    const uint32_t hi = (128u >> 4) | (1u << 14), lbo = (1024u >> 4) << 16;
    const uint32_t wh = wgt >> 4 | lbo, wl = (wgt + part) >> 4 | lbo, xl = act >> 4 | lbo, xh = (act + part) >> 4 | lbo;
    bool ok = ptx::mbar_wait_warp(bar_w, 0u, abort_flag, wait_rounds);
    if (!ok) wait_expired(p.err, abort_flag, kErrFullWait);
    int t = 0;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++t) {
      const int buf = t & 1;
      if (t >= 2 && !ptx::mbar_wait_warp(bar_acc_empty + 8 * buf, (uint32_t)(((t >> 1) - 1) & 1), abort_flag, wait_rounds)) {
        wait_expired(p.err, abort_flag, kErrAccWait);
        break;
      }
      const uint32_t d = tmem_base + (uint32_t)buf * kStemPx;
      for (int term = 0; term < 3 && ok; ++term) {
        if (term < 2) {
          ok = ptx::mbar_wait_warp(bar_full + 8 * term, (uint32_t)(t & 1), abort_flag, wait_rounds);
          if (!ok) {
            wait_expired(p.err, abort_flag, kErrFullWait);
            break;
          }
          ptx::tcgen05_fence_after();
        }
        const uint32_t w_lo = term == 1 ? wl : wh, x_lo = term == 0 ? xl : xh;
        if (ptx::elect_one()) {
          for (int k = 0; k < taps2 / 2; ++k)
            ptx::tcgen05_mma_tf32_lohi<false>(d, w_lo + 128u * k, hi, x_lo + 128u * k, hi, p.idesc, term + k > 0 ? 1u : 0u);
          if (term == 0) ptx::tcgen05_commit(bar_empty);
          if (term == 2) {
            ptx::tcgen05_commit(bar_empty + 8);
            ptx::tcgen05_commit(bar_acc_full + 8 * buf);
          }
        }
        __syncwarp();
      }
    }
  } else if ((warp & 3) < 2) {
    // ------------------------------------------------------------------------------------------------------ epilogue
    const int quarter = warp & 3, half = (warp - 8) >> 2, ch = quarter * 32 + lane;
    const bool ch_ok = ch < p.n_valid;
    const float bias = ch_ok ? __int_as_float(__ldg(p.bias + ch)) : 0.0f;
    pdl_wait();
    int t = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++t) {
      const int buf = t & 1, m0 = tile * kStemPx;
      if (!ptx::mbar_wait_warp(bar_acc_full + 8 * buf, (uint32_t)((t >> 1) & 1), abort_flag, wait_rounds)) {
        wait_expired(p.err, abort_flag, kErrAccWait);
        break;
      }
      ptx::tcgen05_fence_after();
      uint8_t *out = reinterpret_cast<uint8_t *>(p.out) + (size_t)m0 * p.ldc + (size_t)ch * 4;
      epilogue_channels_f32<RELU>(p, tmem_base + (uint32_t)buf * kStemPx + ((uint32_t)(quarter * 32) << 16), out, ch_ok, m0, half, 2, bias, kStemPx);
      ptx::tcgen05_fence_before();
      __syncwarp();
      if (lane == 0 && !p.lose_arrival) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_acc_empty + 8 * buf) : "memory");
    }
  }

  if (threadIdx.x == 0) // the weights' copy has landed, whatever happened
    for (uint32_t i = 0; i < (1u << 20); ++i)
      if (ptx::mbar_try_wait(bar_w, 0u)) break;
  ptx::tcgen05_fence_before();
  __syncthreads();
  if (warp == 10) {
    ptx::tcgen05_fence_after();
    ptx::tcgen05_dealloc(tmem_base, 128u);
  }
}

} // namespace tpucb
