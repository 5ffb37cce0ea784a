// Host planner for the INT8 implicit-GEMM kernel: weight packing, TMA tensor
// maps, tile-shape heuristics and the launch. The geometry follows parseConvParam
// (lib/Dialect/TPU/IR/TPUOperationSupport.cpp:366-428): four independent pads, the
// output size taken from the result type, dilation, optional input zero-insertion.
#pragma once
#include "conv_big.cuh"
#include "conv_stem_f32.cuh"
#include "host_common.h"
#include "mem_kernels.cuh"
#include "per_device.h"

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <cudaTypedefs.h>

namespace tpucb {

struct ConvGeom {
  int n, ic, ih, iw, oc, oh, ow, g, kh, kw, sh, sw, pt, pb, pl, pr, dh, dw, ins_h, ins_w;
};

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*EncodeIm2colFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                   const cuuint64_t *, const cuuint64_t *, const int *, const int *,
                                   cuuint32_t, cuuint32_t, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion,
                                   CUtensorMapFloatOOBfill);

struct TmaApi {
  EncodeTiledFn tiled = nullptr;
  EncodeIm2colFn im2col = nullptr;
  int driver_version = 0;
};

// The driver entry points are fetched through the runtime so that the library carries no
// link-time dependency on the driver library (it must load on machines without a GPU).
inline const TmaApi &tma_api() {
  static TmaApi api = [] {
    TmaApi a;
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    TPUCB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
    TPUCB_CHECK(fn && q == cudaDriverEntryPointSuccess, "cuTensorMapEncodeTiled not available");
    a.tiled = (EncodeTiledFn)fn;
    fn = nullptr;
    TPUCB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &fn, cudaEnableDefault, &q));
    TPUCB_CHECK(fn && q == cudaDriverEntryPointSuccess, "cuTensorMapEncodeIm2col not available");
    a.im2col = (EncodeIm2colFn)fn;
    TPUCB_CUDA(cudaDriverGetVersion(&a.driver_version));
    return a;
  }();
  return api;
}

inline CUtensorMapSwizzle swizzle_for(int BK) {
  return BK == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                   : (BK == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

// tcgen05 instruction descriptor for kind::i8: D = s32 (bits 4-5 = 2), A and B signed
// 8-bit (bits 7-9 and 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
inline uint32_t make_idesc_i8(int M, int N) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}

// kind::f16 with BF16 operands and an fp32 accumulator: D = f32 (bits 4-5 = 1), A and B = BF16 (1)
inline uint32_t make_idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// kind::tf32 with an fp32 accumulator: D = f32 (1), A and B = TF32 (2)
inline uint32_t make_idesc_tf32(int M, int N) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

struct ConvPlan {
  CUtensorMap tmA, tmB;
  ConvGemmParams p;
  dim3 grid;
  size_t smem = 0;
  int ws_tiles = 0;  // split K: tiles of the partial-sum workspace (p.ws, p.ws_count), allocated by the op that owns the plan
  bool bf16 = false; // runs conv_gemm_bf16_kernel (K sizes and pitches in bytes, 2 per element)
  bool tf32 = false; // runs conv_gemm_tf32x3_kernel (fp32 operands, 4 bytes per element; three K passes)
  int ctas = 0;      // runs the kernels of conv_big.cuh with this many CTAs per tile (0: those of conv_gemm_i8.cuh)
  CUtensorMap tmO, tmO2; // ctas > 0: the results, and those of the fused activation or the remainder operand
  bool stem = false; // runs conv_stem_tf32x3_kernel
  StemArgs stem_args;
  int box_px() const { return ctas > 1 ? p.m_tile / ctas : p.m_tile; } // pixels per copy of the activations
  CUtensorMap tmA2, tmB2;           // tf32: remainder parts of the activations and of the weights
  const float *split_src = nullptr; // tf32: the fp32 input, whose remainder is written to split_lo before the launch
  float *split_lo = nullptr;
  size_t split_nvec = 0;
  bool use_patch = false;
  PatchArgs patch;
  int8_t *patch_buf = nullptr; // scratch: expanded patch matrix [M][kp]
  size_t patch_bytes = 0;
  bool use_repack = false; // row windows: the input's rows are copied into the window layout first
  RepackArgs repack;
  const int8_t *in = nullptr;
  double ops = 0, bytes = 0; // algorithmic work of one launch
};

// K block width in bytes for `k_bytes` of K per tap. The main loop's time follows the NUMBER of K blocks (a block
// costs a barrier round trip and a copy issue whatever its width), so the fewest blocks win and, among equal counts,
// the narrower block (less zero padding through the tensor pipe): 96 bytes -> one 128-byte block, not three of 32.
inline int pick_bk(int k_bytes) {
  int best = 128, best_blocks = 1 << 30;
  for (int bk : {128, 64, 32}) {
    int blocks = (k_bytes + bk - 1) / bk;
    if (blocks <= best_blocks) {
      best_blocks = blocks;
      best = bk;
    }
  }
  return best;
}

// One output channel's filter, [channels][taps] -> [taps][pitch] of T: converted in one sweep (which the compiler
// vectorises), then the taps are told apart; `line` holds channels * taps values.
template <class T, class Convert>
inline void pack_filter(const float *w, int channels, int taps, T *out, size_t pitch, T *line, Convert convert) {
  T *to = taps == 1 ? out : line;
  const size_t n = (size_t)channels * taps;
  for (size_t i = 0; i < n; ++i) to[i] = convert(w[i]);
  if (taps > 1)
    for (int t = 0; t < taps; ++t)
      for (int c = 0; c < channels; ++c) out[t * pitch + c] = line[(size_t)c * taps + t];
}

// Rows of the packed weights: whole blocks of 32 channels, in the order of packed_row (`natural`: of the channels, for conv_big.cuh).
inline size_t packed_rows(int oc_pad) { return (size_t)(oc_pad + 31) / 32 * 32; }

// Pack OIHW fp32 weights (integer-valued) to int8 [rows][taps][cin_pad] for the im2col
// path, or [rows][1][kp] with K order (r, s, c) for the patch path. For grouped
// convolution the caller passes one group's slice.
inline std::vector<int8_t> pack_conv_weights(const float *w, int oc, int icg, int kh, int kw,
                                             int oc_pad, int cin_pad, bool patch, int kp, bool natural = false) {
  const int taps = kh * kw;
  const size_t row = patch ? kp : (size_t)taps * cin_pad, pitch = patch ? icg : cin_pad;
  std::vector<int8_t> out(packed_rows(oc_pad) * row, 0), line((size_t)icg * taps);
  for (int o = 0; o < oc; ++o)
    pack_filter(w + (size_t)o * icg * taps, icg, taps, out.data() + (natural ? o : packed_row(o)) * row, pitch, line.data(), [](float v) { return (int8_t)(int)v; });
  return out;
}

// BF16 weights [rows][tap][cin_pad] as 16-bit patterns (the values of a BF16 graph's filter are
// BF16-representable floats: the upper 16 bits are the value), returned as bytes
inline std::vector<int8_t> pack_conv_weights_bf16(const float *w, int oc, int icg, int kh, int kw, int oc_pad,
                                                  int cin_pad, bool natural) {
  const int taps = kh * kw;
  const size_t row = (size_t)taps * cin_pad;
  std::vector<int8_t> bytes(packed_rows(oc_pad) * row * 2, 0);
  std::vector<uint16_t> line((size_t)icg * taps);
  for (int o = 0; o < oc; ++o)
    pack_filter(w + (size_t)o * icg * taps, icg, taps, reinterpret_cast<uint16_t *>(bytes.data()) + (natural ? o : packed_row(o)) * row, cin_pad, line.data(),
                [](float v) { return (uint16_t)(f32_bits(v) >> 16); });
  return bytes;
}

// fp32 weights for the TF32 x 3 convolution, K-major [rows][tap][cin_pad] as bytes: part 0 = the upper 19 bits of
// every word, part 1 = the exact remainder.
inline std::vector<int8_t> pack_conv_weights_tf32(const float *w, int oc, int icg, int kh, int kw, int oc_pad, int cin_pad,
                                                  int part, bool natural) {
  const int taps = kh * kw;
  std::vector<float> out(packed_rows(oc_pad) * taps * cin_pad, 0.0f);
  for (int o = 0; o < oc; ++o)
    for (int c = 0; c < icg; ++c)
      for (int r = 0; r < kh; ++r)
        for (int s = 0; s < kw; ++s) {
          const float v = w[(((size_t)o * icg + c) * kh + r) * kw + s];
          const float hi = bits_f32(f32_bits(v) & 0xffffe000u);
          out[((size_t)(natural ? o : packed_row(o)) * taps + (r * kw + s)) * cin_pad + c] = part == 0 ? hi : v - hi;
        }
  std::vector<int8_t> bytes(out.size() * 4);
  std::memcpy(bytes.data(), out.data(), bytes.size());
  return bytes;
}

// the same for the patch matrix of an fp32 image stem: four channel slots per tap, k = tap * 4 + c
inline std::vector<int8_t> pack_patch_weights_tf32(const float *w, const ConvGeom &g, int oc_pad, int part, bool natural) {
  const int kp = g.kh * g.kw * 4;
  std::vector<float> out(packed_rows(oc_pad) * kp, 0.0f);
  for (int o = 0; o < g.oc; ++o)
    for (int c = 0; c < g.ic; ++c)
      for (int t = 0; t < g.kh * g.kw; ++t) {
        const float v = w[((size_t)o * g.ic + c) * g.kh * g.kw + t], hi = bits_f32(f32_bits(v) & 0xffffe000u);
        out[(size_t)(natural ? o : packed_row(o)) * kp + t * 4 + c] = part == 0 ? hi : v - hi;
      }
  std::vector<int8_t> bytes(out.size() * 4);
  std::memcpy(bytes.data(), out.data(), bytes.size());
  return bytes;
}

// and for the stem kernel: [high parts, remainders][taps, even][64 channels][4]
inline std::vector<int8_t> pack_stem_weights_tf32(const float *w, const ConvGeom &g) {
  const int taps = g.kh * g.kw, taps2 = (taps + 1) / 2 * 2;
  std::vector<float> out((size_t)2 * taps2 * 64 * 4, 0.0f);
  for (int o = 0; o < g.oc; ++o)
    for (int c = 0; c < g.ic; ++c)
      for (int t = 0; t < taps; ++t) {
        const float v = w[((size_t)o * g.ic + c) * taps + t], hi = bits_f32(f32_bits(v) & 0xffffe000u);
        out[((size_t)t * 64 + o) * 4 + c] = hi;
        out[((size_t)(taps2 + t) * 64 + o) * 4 + c] = v - hi;
      }
  std::vector<int8_t> bytes(out.size() * 4);
  std::memcpy(bytes.data(), out.data(), bytes.size());
  return bytes;
}

inline void encode_weight_map(CUtensorMap *tm, const int8_t *d_w, int oc_pad, int taps, int k_inner,
                              int BK, int BN) {
  cuuint64_t dims[3] = {(cuuint64_t)k_inner, (cuuint64_t)taps, (cuuint64_t)packed_rows(oc_pad)};
  cuuint64_t strides[2] = {(cuuint64_t)k_inner, (cuuint64_t)k_inner * taps};
  cuuint32_t box[3] = {(cuuint32_t)BK, 1, (cuuint32_t)BN};
  cuuint32_t es[3] = {1, 1, 1};
  CUresult r = tma_api().tiled(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, (void *)d_w, dims, strides, box,
                               es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(BK),
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TPUCB_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled(weights) failed: %d", (int)r);
}

inline void encode_matrix_map(CUtensorMap *tm, const int8_t *d_a, int rows, int k_inner, int ld,
                              int BK, int tile_rows) {
  cuuint64_t dims[2] = {(cuuint64_t)k_inner, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)tile_rows};
  cuuint32_t es[2] = {1, 1};
  CUresult r = tma_api().tiled(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void *)d_a, dims, strides, box,
                               es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(BK),
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TPUCB_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled(matrix) failed: %d", (int)r);
}

// Drivers up to CUDA 13.1 encode im2col maps of tensors smaller than 128 KiB with a flag (bit 21 of the second 64-bit word)
// that makes the load misbehave; the same correction is applied by NVIDIA's open-source CUTLASS when it builds these maps.
inline void fix_small_im2col_map(CUtensorMap *tm, size_t tensor_bytes) {
  if (tma_api().driver_version <= 13010 && tensor_bytes < 131072) reinterpret_cast<uint64_t *>(tm)[1] &= ~(1ull << 21);
}

inline void encode_im2col_map(CUtensorMap *tm, const int8_t *d_in, const ConvGeom &g, int cp,
                              int BK, int tile_rows) {
  cuuint64_t dims[4] = {(cuuint64_t)cp, (cuuint64_t)g.iw, (cuuint64_t)g.ih, (cuuint64_t)g.n};
  cuuint64_t strides[3] = {(cuuint64_t)cp, (cuuint64_t)cp * g.iw, (cuuint64_t)cp * g.iw * g.ih};
  // Base-pixel bounding box: lower corner = -pad_lo, upper corner chosen so that the number
  // of base positions along each axis equals the op's output extent:
  //   (extent + upper - lower - 1) / stride + 1 == out
  int lower[2] = {-g.pl, -g.pt};
  // Textbook value: pad_hi - (k - 1) * dilation. When the op's output extent does not follow
  // from its pads by the usual formula (the result type rules), use the tight value instead.
  int upper[2] = {g.pr - (g.kw - 1) * g.dw, g.pb - (g.kh - 1) * g.dh};
  if ((g.iw + upper[0] - lower[0] - 1) / g.sw + 1 != g.ow)
    upper[0] = (g.ow - 1) * g.sw + 1 - g.iw - g.pl;
  if ((g.ih + upper[1] - lower[1] - 1) / g.sh + 1 != g.oh)
    upper[1] = (g.oh - 1) * g.sh + 1 - g.ih - g.pt;
  cuuint32_t es[4] = {1, (cuuint32_t)g.sw, (cuuint32_t)g.sh, 1};
  CUresult r = tma_api().im2col(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void *)d_in, dims, strides,
                                lower, upper, (cuuint32_t)BK, (cuuint32_t)tile_rows, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                swizzle_for(BK), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TPUCB_CHECK(r == CUDA_SUCCESS,
              "cuTensorMapEncodeIm2col failed: %d (iw=%d ih=%d lower=%d,%d upper=%d,%d)", (int)r,
              g.iw, g.ih, lower[0], lower[1], upper[0], upper[1]);
  fix_small_im2col_map(tm, (size_t)cp * g.iw * g.ih * g.n);
}

// Few-channel convolutions (image stems) as row windows. The input is stored as zero-padded NHWC rows with a pixel pitch of
// P = 4, 8 or 16 bytes, so that the taps of one filter row of one output pixel are one contiguous window. G neighbouring
// output pixels form one row of the implicit GEMM: their windows overlap, so ONE window of (G - 1) strides more serves
// all of them, against G copies of the filter shifted by one output stride each, which fill the 128 rows of the tensor
// core's weight operand (64 output channels: G = 2, 32: G = 4) instead of zeros. G also makes the windows start on the 16-byte
// boundaries that a tensor map needs. An im2col-mode tensor map whose "width" is the pixel group (stride G * sw * P, window
// bytes as the "channels", overlapping) then brings the windows of a whole tile in one copy per filter row.
struct WindowPlan {
  int P = 0;      // bytes per input pixel
  int G = 1;      // output pixels per GEMM row
  int win = 0;    // window bytes that hold taps
  int wphys = 0;  // pixels per stored row: pl zeros, the row, zeros
};
inline bool window_plan_for(const ConvGeom &g, int es, int oc_pad, WindowPlan *out) {
  if (g.g != 1 || g.ins_h || g.ins_w || (g.kh == 1 && g.kw == 1) || g.ic * es > 16) return false;
  if (g.sh > 8 || g.pt > 127 || g.pb > 127 || (g.kh - 1) * g.dh > 127) return false;
  double best = 0;
  bool found = false;
  for (int G : {4, 2, 1})
    for (int P : {4, 8, 16}) {
      const int win = ((G - 1) * g.sw + (g.kw - 1) * g.dw + 1) * P;
      if (P / es < g.ic || (G > 1 && (oc_pad > 128 / G || g.ow % G)) || G * g.sw * P % 16 || win > 128) continue;
      const double cost = (double)((win + 31) / 32) / G; // tensor-core steps per output pixel and filter row
      if (found && cost >= best) continue;
      found = true;
      best = cost;
      const int bk = win <= 32 ? 32 : (win <= 64 ? 64 : 128);
      int wphys = ((g.ow / G - 1) * G * g.sw * P + bk + P - 1) / P; // the last window, with its padding, stays inside the row
      if (wphys < g.pl + g.iw) wphys = g.pl + g.iw;
      while (wphys * P % 16) ++wphys;
      out->P = P; out->G = G; out->win = win; out->wphys = wphys;
    }
  return found;
}

// Weights of the window form: rows [G][128 / G channels] (one row per channel for G = 1), per filter row BK bytes.
inline std::vector<int8_t> pack_window_weights(const float *w, const ConvGeom &g, const WindowPlan &wp, int rows, int BK, bool bf16) {
  const int es = bf16 ? 2 : 1, slot = 128 / wp.G;
  std::vector<int8_t> out((size_t)rows * g.kh * BK, 0);
  for (int j = 0; j < wp.G; ++j)
    for (int o = 0; o < g.oc; ++o)
      for (int c = 0; c < g.ic; ++c)
        for (int r = 0; r < g.kh; ++r)
          for (int s = 0; s < g.kw; ++s) {
            const float v = w[(((size_t)o * g.ic + c) * g.kh + r) * g.kw + s];
            int8_t *at = out.data() + ((size_t)packed_row(j * slot + o) * g.kh + r) * BK + (size_t)(j * g.sw + s * g.dw) * wp.P + c * es;
            if (bf16) {
              const uint16_t h = (uint16_t)(f32_bits(v) >> 16);
              std::memcpy(at, &h, 2);
            } else {
              *at = (int8_t)(int)v;
            }
          }
  return out;
}

inline void encode_window_map(CUtensorMap *tm, const void *d_in, const ConvGeom &g, const WindowPlan &wp, int BK, int tile_rows) {
  const cuuint64_t row = (cuuint64_t)wp.wphys * wp.P;
  cuuint64_t dims[4] = {(cuuint64_t)BK, (cuuint64_t)(g.ow / wp.G), (cuuint64_t)g.ih, (cuuint64_t)g.n};
  cuuint64_t strides[3] = {(cuuint64_t)wp.G * g.sw * wp.P, row, row * g.ih};
  int lower[2] = {0, -g.pt}, upper[2] = {0, (g.oh - 1) * g.sh + 1 - g.ih - g.pt};
  cuuint32_t es[4] = {1, 1, (cuuint32_t)g.sh, 1};
  CUresult r = tma_api().im2col(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void *)d_in, dims, strides, lower, upper, (cuuint32_t)BK,
                                (cuuint32_t)tile_rows, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(BK),
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TPUCB_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeIm2col(row windows) failed: %d", (int)r);
  fix_small_im2col_map(tm, (size_t)row * g.ih * g.n);
}

// Maps of the tensors that the kernels of conv_big.cuh write: 32 pixels x 128 bytes per store, clipped to the valid
// channels and the last pixel.
inline void encode_out_maps(ConvPlan &pl) {
  if (pl.ctas == 0) return;
  const int es = pl.tf32 ? 4 : (pl.bf16 ? 2 : 1);
  for (int k = 0; k < 2; ++k) {
    int8_t *to = k ? pl.p.out2 : pl.p.out;
    cuuint64_t dims[2] = {(cuuint64_t)pl.p.n_valid * es, (cuuint64_t)pl.p.M_total};
    cuuint64_t strides[1] = {(cuuint64_t)pl.p.ldc};
    cuuint32_t box[2] = {128, 32}, one[2] = {1, 1};
    CUresult r = tma_api().tiled(k ? &pl.tmO2 : &pl.tmO, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, to ? to : pl.p.out, dims, strides, box, one,
                                 CU_TENSOR_MAP_INTERLEAVE_NONE, pl.tf32 ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B,
                                 CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    TPUCB_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled(results) failed: %d", (int)r);
  }
}

// Whether a plan runs on the kernels of conv_big.cuh, and in which form: CTAs per tile (one: 128 channels, two: 256) and
// pixels per tile.
inline bool finish_big_plan(ConvPlan &pl, int rows, int taps, int oc_pad, int sm_count) {
  ConvGemmParams &p = pl.p;
  const int mode = conv_big_mode(), kind = pl.tf32 ? 2 : (pl.bf16 ? 1 : 0);
  if (mode == 0 || p.group > 1 || p.c_off || oc_pad % 16 || (kind == 0 && !p.fq && !(p.fastq & 1))) return false;
  const int k_iters = taps * p.c_chunks * (kind == 2 ? 3 : 1);
  int ctas = mode > 1 ? mode / 1000 : 0, px = mode % 1000;
  auto tiles_of = [&](int c, int n) { return (long long)((rows + n - 1) / n) * ((oc_pad + 128 * c - 1) / (128 * c)); };
  if (mode == 1 && kind < 2) {
    // Launches of 1.3 tiles of 128 x 256 per SM and more, whose K is long enough that its loop counts and not the epilogue, which
    // the kernels of conv_gemm_i8.cuh do better (INT8 from 8 K blocks, BF16 from 2); pairs where the loop is nearly everything.
    // us alone / with three launches in flight, there -> here:
    //   INT8, 256 images: 3x3 256 channels 14x14 25.4 / 24.6 -> 22.4 / 21.3 (pair), 128 at 28x28 27.3 / 28.0 -> 24.3 / 25.4, 512 at
    //     7x7 28.6 / 22.6 -> 25.9 / 20.1, 64 at 56x56 52.0 / 50.5 -> 46.4 / 45.1; 1x1 1024 -> 256 14.2 / 15.7 -> 13.0 / 15.0;
    //     large ones: 32 x 512 x 56 x 56 183 / 180 -> 158 / 155 (single), 140 / 141 (pair);
    //     not: 1x1 512 -> 2048 (4 blocks) 18.1 / 16.6 against 20.1 / 17.9, 64 -> 256 58 / 53 against 62 / 59;
    //   BF16, 128 images: 3x3 256 at 14x14 28.7 / 23.6 -> 27.2 / 21.5, 512 at 7x7 30.3 / 22.5 -> 26.5 / 20.0; 1x1 256 -> 1024 18.6 /
    //     18.4 -> 16.9 / 16.3, 128 -> 512 25.3 / 24.6 -> 24.1 / 23.0; not 64 -> 256 43.7 / 40.4 against 45.6 / 39.5;
    //   fewer tiles: INT8, 64 images, 128 at 28x28 (196) 10.9 / 8.5 against 11.0 / 8.6, 256 at 14x14 (98) 10.9 / 6.7 against 10.5 /
    //     6.7; tiles of 192 pixels 9.2 / 8.0: faster alone, slower in flight.
    if (oc_pad <= 64 || tiles_of(1, 256) * 10 < 13LL * sm_count || k_iters < (kind == 0 ? 8 : 2)) return false;
    px = 256;
    ctas = oc_pad > 128 && k_iters >= 16 && tiles_of(2, 256) >= sm_count ? 2 : 1;
  } else if (mode == 1) {
    // fp32 runs alone (calibration, the tuner), so whole waves count: clocks per K block of a wave, as measured (3x3 256
    // channels at 14x14 and 128 at 28x28, 64 images: 85.6 -> 66.2 us and 79.0 -> 70.8; 1x1 1024 -> 256 55.9 -> 46.1, 256 -> 1024
    // 40.5 -> 35.8; not: 3x3 512 at 7x7, one tile per SM there, 106 against 118).
    if (oc_pad <= 64) return false;
    const long long there = (tiles_of(1, 128) + sm_count - 1) / sm_count;
    double best = there <= 1 ? 466.0 : 376.0 * there;
    for (int c = 1; c <= (k_iters >= 16 ? 2 : 1); ++c)
      for (int n = 128; n <= 256; n += 64) {
        const long long slots = sm_count / c, waves = (tiles_of(c, n) + slots - 1) / slots;
        const double cost = waves * (c == 1 ? std::max(520.0, 2.5 * n) : std::max(530.0, 2.37 * n));
        if (cost > 0.97 * best && (ctas == 0 || cost > best)) continue;
        best = cost;
        ctas = c;
        px = n;
      }
    if (ctas == 0) return false;
  }
  const size_t stage = (size_t)(128 + px / ctas) * p.BK, fixed = 1024 + kBigHeader + kBigStaging[kind];
  int stages = (int)std::min<size_t>(kMaxStages, (227 * 1024 - fixed) / stage);
  if (stages < 2) return false;
  pl.ctas = ctas;
  p.dual = 0;
  p.w_resident = 0;
  p.split_k = 1;
  p.k_per = taps * p.c_chunks;
  p.BN = 128;
  p.n_valid = oc_pad;
  p.tmem_cols = 512;
  p.m_tile = px;
  p.stages = stages;
  const int M = 128 * ctas;
  p.idesc = kind == 2 ? make_idesc_tf32(M, px) : (kind == 1 ? make_idesc_bf16(M, px) : make_idesc_i8(M, px));
  const long long tiles = (long long)((rows + px - 1) / px) * ((oc_pad + M - 1) / M);
  pl.grid = dim3((unsigned)(ctas * std::min<long long>(tiles, sm_count / ctas)), 1, 1);
  // (More than half of an SM's shared memory in any case: two CTAs of these kernels on one SM would wait for each other's
  // tensor memory.)
  pl.smem = std::max<size_t>(fixed + stages * stage, 120 * 1024);
  return true;
}

// Build the launch plan for one GEMM-shaped problem.
//   rows       implicit-GEMM M
//   k_inner    K bytes per tap (padded input channels, or the whole K in matrix mode)
//   oc_pad     padded output channels (multiple of 16)
inline void finish_plan(ConvPlan &pl, int rows, int taps, int k_inner, int oc_pad, int sm_count, bool may_be_big = false) {
  ConvGemmParams &p = pl.p;
  p.M_total = rows;
  p.BK = pick_bk(k_inner);
  p.c_chunks = (k_inner + p.BK - 1) / p.BK;
  p.ksteps = p.c_chunks == 1 ? (k_inner + 31) / 32 : p.BK / 32;
  if (may_be_big && finish_big_plan(pl, rows, taps, oc_pad, sm_count)) return;
  // Dual mode: layers with at most 64 output channels would leave half of the TMEM lanes (and half of
  // the epilogue warps) idle; they run 256-pixel tiles instead (see the kernel). Not combined with
  // pixel groups, which fill them.
  {
    // ... unless the whole weight set is small enough to stay resident in plain mode, which feeds
    // fewer bytes per pixel (measured faster for the 1x1 layers with 64 outputs).
    const size_t w_plain = (size_t)taps * p.c_chunks * 128 * p.BK;
    const bool plain_resident = w_plain <= 48 * 1024 && 113 * 1024 - kSmemHeader - 1024 - w_plain >= 3 * (size_t)128 * p.BK;
    p.dual = (oc_pad <= 64 && p.group <= 1 && rows > 128 && !plain_resident && !pl.tf32) ? 1 : 0;
  }
  // Transposed product: the channel tile is the tensor core's M (128 TMEM lanes, rows past the
  // padded channel count are zero-filled by TMA), the pixel tile its N (128 TMEM columns), and
  // the accumulator is double-buffered: 256 TMEM columns.
  const int bn = 128;
  p.BN = bn;
  p.n_valid = oc_pad;
  p.tmem_cols = 256;
  const int k_iters = taps * p.c_chunks;
  const int n_tiles = (oc_pad + bn - 1) / bn;
  // A launch of few tiles takes half tiles: twice the CTAs, each with half the epilogue and three quarters of the bytes per K
  // block. Up to a third of the SMs; us alone / with three modules in flight, no half tiles -> by this rule: ResNet-50 INT8 batch 1
  // 260.0 / 110.8 -> 240.0 / 98.4, 4 319.6 / 131.7 -> 285.5 / 122.5, 8 354.2 / 159.1 -> 315.2 / 155.7, 19 398.7 / 232.6 -> 385.4 / 229.0, BF16 batch
  // 2 514.4 / 191.2 -> 435.0 / 162.2, 8 550.0 / 230.1 -> 486.0 / 212.1, YOLOv4-style batch 1 855.5 / 357.1 -> 740.1 / 322.9. With more, launches
  // of other streams that would have run beside this one no longer fit. Up to half of the SMs: alone faster, in flight level or
  // slower: INT8 batch 4 285.0 / 123.1, 8 312.8 / 156.0, 19 374.8 / 230.4, BF16 batch 8 483.3 / 215.7, 32 771.0 / 526.5 -> 743.4 / 530.1 (a layer by
  // itself, 7 x 23 x 23, 5x5 of 72 -> 200 channels, 58 tiles, 15.1 / 5.2 -> 10.9 / 4.8). All that have the SMs for it: 4 284.4 / 128.1, 8 311.4 /
  // 164.3, 19 373.0 / 247.3, BF16 8 465.5 / 227.4, 32 717.4 / 548.5. fp32 runs alone and has nothing to gain from another line: batch
  // 4 1449 (none 1488, half of the SMs 1441, all 1446), 16 1945 (1954, 1937, 1964), 30 2627 (2629, 2627, 2678), 64 4500 (4502, 4503,
  // 4544). Quarter tiles gained nothing more.
  p.m_tile = p.dual ? 256 : 128;
  if (!p.dual && (rows + 127) / 128 * n_tiles * 3 <= sm_count) p.m_tile = 64;
  const int m_tiles = (rows + p.m_tile - 1) / p.m_tile;
  const int mma_n = std::min(p.m_tile, 128);
  p.idesc = pl.tf32 ? make_idesc_tf32(128, mma_n) : (pl.bf16 ? make_idesc_bf16(128, mma_n) : make_idesc_i8(128, mma_n));
  const long long total_tiles = (long long)m_tiles * n_tiles;
  const size_t a_bytes = (size_t)p.m_tile * p.BK, b_bytes = (size_t)(p.dual ? 192 : bn) * p.BK;
  const size_t w_all = (size_t)k_iters * b_bytes;
  // Weight-resident mode: when all K blocks of one channel tile's weights fit in 48 KB beside a useful
  // ring of activation tiles (two CTAs per SM are kept), a CTA loads them once and streams only
  // activations, which halves the bytes that have to reach shared memory per MAC. Larger weight
  // sets would force one CTA per SM, which measured slower than re-fetching the weights from L2.
  const int ctas_per_sm = 2;
  // (An fp32 launch of at most one CTA per SM takes all of the shared memory: ResNet-50 at batch 30 alone, as calibration and
  // the tuner run it, 3455 -> 3377 us. Launches of other streams no longer fit beside it, three modules in flight 2474 ->
  // 2653, which is why INT8 and BF16 launches leave half.)
  const size_t budget = (pl.tf32 && total_tiles <= sm_count ? 220 : 113) * 1024;
  // (Pixel groups have small activation tiles: up to 60 KB of weights leave them four stages.)
  p.w_resident = (!pl.tf32 && total_tiles >= 2LL * n_tiles && w_all <= (p.group > 1 ? 60 : 48) * 1024 &&
                  budget - kSmemHeader - 1024 - w_all >= (p.group > 1 ? 4 : 3) * a_bytes) ? 1 : 0;
  const size_t stage_bytes = p.w_resident ? a_bytes : a_bytes + b_bytes;
  const size_t ring_budget = budget - kSmemHeader - 1024 - (p.w_resident ? w_all : 0);
  int stages = (int)(ring_budget / stage_bytes);
  if (stages < 2) stages = 2;
  if (stages > kMaxStages) stages = kMaxStages;
  int grid = ctas_per_sm * sm_count;
  if (grid > total_tiles) grid = (int)total_tiles;
  if (p.w_resident) {
    grid = grid / n_tiles * n_tiles; // a CTA's channel tile must not change
    if (grid < n_tiles) grid = n_tiles;
  }
  // Split K: a launch with fewer tiles than SMs and a long K gives each tile to several CTAs (ConvGemmParams::split_k): at
  // least six K blocks per CTA, at most sixteen CTAs per tile, no more CTAs than SMs. A K block takes 0.21 us of a CTA that
  // has its SM to itself (0.25 for a tile of 128 pixels). The exchange through global memory (reductions, fence, count, read
  // back) takes 3.4 us for a few CTAs and 4.9 from 75 on (tiles of 128 pixels: 8.5 from 100 on, twice the partial sums).
  // Split where that pays by half a microsecond; us alone and with three streams in flight, unsplit -> split:
  //   3x3, 512 channels, 7x7: N = 1 10.6 / 4.9 -> 8.0 / 4.1 (6 parts), 4 10.7 / 4.9 -> 9.3 / 4.5, 8 10.8 / 4.9 -> 10.0 / 4.9 (5); not
  //   split: 12 11.2 / 4.9 against 10.8 / 5.0 (3);
  //   3x3, 512 -> 1024 channels, 13x13: N = 1 10.8 / 4.9 -> 9.8 / 4.9 (6); not split: 2 11.1 / 4.9 against 10.9 / 5.5 (3);
  //   3x3, 1024 channels, 5x5: N = 2 18.4 / 7.6 -> 9.2 / 4.5 (12), 8 18.5 / 7.6 -> 12.3 / 5.6 (4).
  // Two CTAs per SM were a loss wherever other work fills the gaps (5x5, 64 -> 128 channels, 7 x 45 x 45, 222 CTAs: 16.1 us
  // against 12.7 unsplit, three streams at once 9.8 against 5.3). The weights are then not kept resident (a CTA needs only
  // its own K range once).
  p.split_k = 1;
  p.k_per = k_iters;
  if (conv_split_k_enabled() && !pl.tf32 && !pl.bf16 && !p.dual) {
    const int want = (int)std::min<long long>(std::min(16, k_iters / 6), sm_count / total_tiles);
    if (want >= 2) {
      const int per = (k_iters + want - 1) / want, parts = (k_iters + per - 1) / per;
      const double ctas = (double)total_tiles * parts;
      const double block = p.m_tile == 64 ? 0.21 : 0.25;
      const double exchange = 3.4 + (p.m_tile == 64 ? 0.02 * std::min(ctas, 75.0) : 0.051 * std::min(ctas, 100.0));
      if (block * (k_iters - per) > exchange + 0.5) {
        p.k_per = per;
        p.split_k = parts;
      }
    }
  }
  if (p.split_k > 1) {
    if (p.w_resident) {
      p.w_resident = 0;
      stages = (int)((budget - kSmemHeader - 1024) / (a_bytes + b_bytes));
      if (stages < 2) stages = 2;
      if (stages > kMaxStages) stages = kMaxStages;
    }
    grid = (int)total_tiles * p.split_k;
    pl.ws_tiles = (int)total_tiles;
  }
  const size_t stage_bytes_final = p.w_resident ? a_bytes : a_bytes + b_bytes;
  const long long iters_per_cta = p.split_k > 1 ? p.k_per
                                                : ((total_tiles + grid - 1) / grid) * k_iters * (pl.tf32 ? 3 : 1);
  if (stages > iters_per_cta) stages = (int)iters_per_cta;
  if (stages < 1) stages = 1;
  p.stages = stages;
  pl.smem = kSmemHeader + 1024 + (p.w_resident ? w_all : 0) + stages * stage_bytes_final;
  pl.grid = dim3((unsigned)grid, 1, 1);
}

// ---- pixel pairs -------------------------------------------------------------------------------------------------------
// A stride-1 layer with at most 64 output channels would use half of the tensor core's rows. In NHWC memory two neighbouring
// pixels of cp channels are one pixel of 2 cp channels, on both sides, so the layer is also a convolution of half the width
// from 2 cp to 2 cp channels, whose filter holds the original one twice, the second time a pixel (half a channel block)
// further. The rows fill up, tile rows are twice as long, and of a 3x3 filter's nine taps of twice the channels a third meets
// only zero weights.
struct DenseLayer {
  ConvGeom g; // g.ic = in_cp and g.oc = out_cp once paired
  int in_cp, out_cp;
  const float *w;         // OIHW: the caller's filter, or `own` once paired
  std::vector<float> own;
  std::vector<float> bias, mult, rshift; // per channel
  bool paired = false;
};
inline bool pair_applies(const ConvGeom &g, int in_cp, int out_cp, int es) {
  if (g.sh != 1 || g.sw != 1 || out_cp > 64 || g.iw % 2 || g.ow % 2 || g.ow < 4) return false;
  // 1x1: the weights double (half of them zeros) and should still stay in shared memory
  if (g.kw == 1) return g.kh == 1 && g.pl == 0 && g.pt == 0 && g.oh == g.ih && g.ow == g.iw && in_cp * es <= 128;
  return g.pl <= 127;
}
inline void pair_layer(DenseLayer &d) {
  const ConvGeom g = d.g;
  const int pl2 = (g.pl + 1) / 2;
  const int kw2 = (1 + (g.kw - 1) * g.dw - g.pl + 2 * pl2) / 2 + 1; // the last input pixel's pair, counted from the first
  const int ic2 = 2 * d.in_cp, oc2 = 2 * d.out_cp;
  std::vector<float> w((size_t)oc2 * ic2 * g.kh * kw2, 0.0f);
  for (int e = 0; e < 2; ++e)
    for (int o = 0; o < g.oc; ++o)
      for (int c = 0; c < g.ic; ++c)
        for (int r = 0; r < g.kh; ++r)
          for (int s = 0; s < g.kw; ++s) {
            const int t = e + s * g.dw - g.pl + 2 * pl2; // input pixel counted from the first of the leftmost pair
            w[(((size_t)(e * d.out_cp + o) * ic2 + (t % 2) * d.in_cp + c) * g.kh + r) * kw2 + t / 2] =
                d.w[(((size_t)o * g.ic + c) * g.kh + r) * g.kw + s];
          }
  auto twice = [&](std::vector<float> &v) {
    std::vector<float> o((size_t)oc2, 0.0f);
    for (size_t i = 0; i < v.size(); ++i) o[i] = o[d.out_cp + i] = v[i];
    v = o;
  };
  twice(d.bias);
  if (!d.mult.empty()) {
    twice(d.mult);
    twice(d.rshift);
  }
  d.own = std::move(w);
  d.w = d.own.data();
  d.g.ic = ic2; d.g.oc = oc2; d.g.iw /= 2; d.g.ow /= 2; d.g.kw = kw2; d.g.dw = 1; d.g.pl = pl2;
  d.g.pr = d.g.ow - d.g.iw - pl2 + kw2 - 1;
  d.in_cp = ic2;
  d.out_cp = oc2;
  d.paired = true;
}

// How a plan runs, in words (tpucb_interp_get_op_form).
inline std::string conv_form(const ConvPlan &pl) {
  const ConvGemmParams &p = pl.p;
  const bool floating = p.fq && p.split_k <= 1;
  return std::string("tiles=") + (pl.stem ? "stem" : (pl.ctas > 0 ? "big" : "small")) + " ctas=" + std::to_string(std::max(1, pl.ctas)) +
         " pixels=" + std::to_string(pl.stem ? kStemPx : p.m_tile) + " split_k=" + std::to_string(std::max(1, p.split_k)) +
         " requant=" + (pl.bf16 || pl.tf32 ? "none" : (floating ? "float" : (p.fastq & 1 ? "integer" : "wide")));
}

// The tensor-core kernel of a plan, as a constant that `use` gets.
template <auto K> struct KernelConstant {
  static constexpr auto value = K;
};
template <class Use> inline void with_conv_kernel(const ConvPlan &pl, Use use) {
  const ConvGemmParams &p = pl.p;
  if (pl.stem) {
    if (p.act == 1) use(KernelConstant<conv_stem_tf32x3_kernel<true>>());
    else use(KernelConstant<conv_stem_tf32x3_kernel<false>>());
  } else if (pl.ctas > 0) {
    auto by_ctas = [&](auto c) {
      constexpr int C = decltype(c)::value;
      if (pl.tf32) {
        if (p.act == 1) use(KernelConstant<conv_big_tf32x3_kernel<C, 1>>());
        else use(KernelConstant<conv_big_tf32x3_kernel<C, 0>>());
      } else if (pl.bf16) {
        if (p.act == 1) use(KernelConstant<conv_big_kernel<C, 1, 1, 0>>());
        else use(KernelConstant<conv_big_kernel<C, 1, 0, 0>>());
      } else if (p.fq) {
        if (p.act == 1) use(KernelConstant<conv_big_kernel<C, 0, 1, 3>>());
        else if (p.act == 2) use(KernelConstant<conv_big_kernel<C, 0, 2, 3>>());
        else use(KernelConstant<conv_big_kernel<C, 0, 0, 3>>());
      } else {
        if (p.act == 1) use(KernelConstant<conv_big_kernel<C, 0, 1, 1>>());
        else if (p.act == 2) use(KernelConstant<conv_big_kernel<C, 0, 2, 1>>());
        else use(KernelConstant<conv_big_kernel<C, 0, 0, 1>>());
      }
    };
    if (pl.ctas == 2) by_ctas(std::integral_constant<int, 2>());
    else by_ctas(std::integral_constant<int, 1>());
  } else if (pl.tf32) use(KernelConstant<conv_gemm_tf32x3_kernel>());
  else if (pl.bf16 && p.act == 3) use(KernelConstant<conv_gemm_bf16_add_kernel>());
  else if (pl.bf16) use(KernelConstant<conv_gemm_bf16_kernel>());
  else if (p.split_k > 1 && (p.fastq & 1)) use(KernelConstant<conv_gemm_i8_split_kernel<true>>());
  else if (p.split_k > 1) use(KernelConstant<conv_gemm_i8_split_kernel<false>>());
  else if (p.fq && p.act == 1) use(KernelConstant<conv_gemm_i8_fq_kernel<1>>());
  else if (p.fq && p.act == 0) use(KernelConstant<conv_gemm_i8_fq_kernel<0>>());
  else if (p.fq && p.act == 2) use(KernelConstant<conv_gemm_i8_fq_kernel<2>>());
  else if (p.fq) use(KernelConstant<conv_gemm_i8_fq_kernel<3>>());
  else if (!(p.fastq & 1)) use(KernelConstant<conv_gemm_i8_wide_kernel>());
  else use(KernelConstant<conv_gemm_i8_kernel>());
}
// To be called at load for every plan, and again when its activation changes, on the device that will run it: the limit of
// shared memory belongs to a kernel on a device. Only the kernels that are used are set up: the driver loads a kernel when its
// attribute is set, which takes half a millisecond each.
inline void conv_kernel_ready(const ConvPlan &pl) {
  int device = 0;
  TPUCB_CUDA(cudaGetDevice(&device));
  with_conv_kernel(pl, [&](auto k) {
    static OncePerDevice ready; // one of each kernel
    ready.run(device, [] { TPUCB_CUDA(cudaFuncSetAttribute(decltype(k)::value, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024)); });
  });
}

inline void launch_conv_plan(const ConvPlan &pl, cudaStream_t stream, int sm_count) {
  if (pl.use_patch && pl.tf32)
    launch_k(patch_expand_f32_kernel, grid_for((size_t)pl.p.M_total * pl.patch.kp / 4, 256, sm_count), 256, 0, stream,
             reinterpret_cast<const float4 *>(pl.in), reinterpret_cast<float4 *>(pl.patch_buf), reinterpret_cast<float4 *>(pl.split_lo), pl.patch);
  else if (pl.use_patch)
    launch_k(patch_expand_i8_kernel, grid_for((size_t)pl.p.M_total * pl.patch.kp, 256, sm_count), 256, 0, stream, pl.in, pl.patch_buf, pl.patch);
  if (pl.use_repack) {
    const RepackArgs &a = pl.repack;
    const int grid = (int)std::min<size_t>(a.rows, (size_t)sm_count * 8);
    if (a.es == 1) launch_k(window_repack_kernel<uint8_t>, grid, 256, 0, stream, a);
    else launch_k(window_repack_kernel<uint16_t>, grid, 256, 0, stream, a);
  }
  PdlConvScope conv_class; // the tensor-core kernel and its helper passes may start while the predecessor finishes
  if (pl.tf32 && !pl.stem && pl.split_src)
    launch_k(tf32_split_kernel, grid_for(pl.split_nvec, 256, sm_count), 256, 0, stream, reinterpret_cast<const float4 *>(pl.split_src),
             reinterpret_cast<float4 *>(pl.split_lo), pl.split_nvec);
  const int threads = pl.stem ? kStemThreads : (pl.ctas > 0 ? kBigThreads : kConvThreads);
  with_conv_kernel(pl, [&](auto k) {
    constexpr auto kernel = decltype(k)::value;
    typedef std::remove_const_t<decltype(kernel)> Kernel;
    using Map = CUtensorMap;
    auto go = [&](auto &&...args) { launch_k(kernel, pl.grid, threads, pl.smem, stream, args..., pl.p); };
    if constexpr (std::is_invocable_v<Kernel, StemArgs, ConvGemmParams>) go(pl.stem_args);
    else if constexpr (std::is_invocable_v<Kernel, Map, Map, ConvGemmParams>) go(pl.tmA, pl.tmB);
    else if constexpr (std::is_invocable_v<Kernel, Map, Map, Map, Map, Map, Map, ConvGemmParams>) go(pl.tmA, pl.tmB, pl.tmA2, pl.tmB2, pl.tmO, pl.tmO2);
    else if (pl.ctas > 0) go(pl.tmA, pl.tmB, pl.tmO, pl.tmO2);
    else go(pl.tmA, pl.tmB, pl.tmA2, pl.tmB2);
  });
}

} // namespace tpucb
