// fp32 convolution on the tensor cores as three TF32 products, for sm_100a.
//
// x = xh + xl, w = wh + wl (h: the upper 19 bits of the word): x w = xh wh + xl wh + xh wl up to 2^-22 relative. The tensor
// core ignores the low 13 bits, so it reads xh out of x itself; four warps write xl = x - xh of every activation block
// into a second buffer, so no remainder tensor exists in memory. The small terms xl wh + xh wl have an accumulator of their
// own, the large one another, added in the epilogue: a truncated partial sum costs an ulp of ITS accumulator.
//
// An activation BLOCK (a channel chunk of a tile's pixels) is fetched once and stays while its T weight tiles pass by:
//   * tap blocks (stride-1 filters, T = all taps): a box of (rows + halo) x (columns + halo) pixels of one or several images,
//     by one tiled copy whose out-of-range pixels arrive as zeros. The box lies in shared memory as one list of pixels with
//     pitch Pc, and a tap's operand is the same list started (r * Pc + s) pixels later: only the start address of the
//     matrix descriptor changes (the swizzle is a function of the address, so a start on any pixel row is as good as another).
//     The accumulator's columns are then positions of that list; those between the rows of the tile are computed and
//     dropped. With full rows the pitch is IW + max(pl, pr): the right padding of a row is the left padding of the next.
//   * plain blocks (T = 1): a tile of a matrix (1x1), or one tap of an im2col map (strides, row windows).
// The rest is conv_gemm_body's scheme: a producer thread, an MMA-issuing thread, eight epilogue warps, a ring for the weight
// tiles, persistent CTAs (one per SM here), bounded waits.
//
// What bounds it is the shared memory (128 bytes per clock): a 128 x N step reads 32 (128 + N) bytes, and there are three per
// 32 bytes of K. One fetch, one split and one shared-memory write per block instead of per tap, and up to 256 columns per
// product: the 3x3 layers of ResNet-50 at batch 64 take 78-119 us against 98-174 with nine fetches of both parts (190 TFLOP/s
// of fp32 work at best, 145 before), the whole forward 4.90 ms against 5.63. (The same scheme for INT8 and BF16, where
// one product per byte of K leaves the operand reads less to save, measured equal to conv_gemm_body or slower.)
#pragma once
#include "conv_gemm_i8.cuh"

namespace tpucb {

struct TapParams {
  int mode;       // 0 matrix tile, 1 im2col map, 2 tap block
  int blocks;     // activation blocks per tile: K chunks (x taps in mode 1)
  int nb;         // activation buffers
  int act_bytes;  // bytes a block's copy brings
  int act_stride; // bytes between the buffers (a multiple of 1024; mode 2: the tail past the block stays zero)
  int N;          // columns of one product (a multiple of 16, up to 256: the weight operand is then read half as often)
  int acc_bufs;   // accumulators: 2, or 1 for N > 128 (the other CTA of the SM computes during the epilogue)
  int n_used;     // columns that may hold results
  int m_tiles;
  // Launches with few tiles and a long K: `parts` CTAs share a tile, each takes a share of its activation blocks and
  // writes plain sums to its own part of a workspace (p.out; part_bytes apart), which tf32_reduce_kernel adds up in order.
  int parts;
  size_t part_bytes;
  // mode 2: a tile is I images (I > 1: whole images) x R rows x Cw columns of outputs; blocks of Rl x Pc pixels per image
  int R, I, Cw, Pc, Rl, tiles_y, tiles_x, images;
  // Steps of 32 bytes of K at the two ends that meet only zero weights (pixel pairs, see pair_layer): the first filter
  // column uses steps from `skip_first` on, the last one those below `keep_last`, counted over all chunks.
  int skip_first, keep_last;
};

constexpr int kPixTable = 1024; // header offset of the column -> pixel table (int32 x 256)
constexpr int kTransformWarps = 4;
constexpr int kNoPixel = 0x3fffffff;

__global__ void __launch_bounds__(kConvThreads + 32 * kTransformWarps, 1)
conv_tf32x3_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ CUtensorMap tmB2, const ConvGemmParams p, const TapParams q) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (base - raw);
  const uint32_t bar_full = base, bar_empty = base + 64;           // weight ring
  const uint32_t bar_acc_full = base + 128, bar_acc_empty = base + 144;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 168);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 172);
  const uint32_t bar_act_full = base + 192, bar_act_empty = base + 224, bar_lo_full = base + 256; // up to 4 buffers each
  int *pix = reinterpret_cast<int *>(smem + kPixTable);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_tiles = (p.n_valid + 127) / 128;
  int total_tiles = n_tiles * q.m_tiles * q.parts; // with parts, a pixel tile index beyond m_tiles is a further part
  const uint32_t w_tile = 128u * (uint32_t)p.BK, w_bytes = 2u * w_tile;
  const uint32_t act0 = base + kSmemHeader;
  const uint32_t lo0 = act0 + (uint32_t)(q.nb * q.act_stride); // remainder blocks
  const uint32_t ring0 = lo0 + (uint32_t)(q.nb * q.act_stride);
  const int taps = q.mode == 2 ? p.kh * p.kw : 1; // weight tiles per block
  const int wait_rounds = p.wait_rounds > 0 ? p.wait_rounds : 1024;
  const int walk_m0 = (int)blockIdx.x / n_tiles, walk_n0 = (int)blockIdx.x % n_tiles;
  const int walk_dm = (int)gridDim.x / n_tiles, walk_dn = (int)gridDim.x % n_tiles;
  const uint32_t half_cols = q.acc_bufs == 2 ? 128u : 256u;          // columns of an accumulator
  const uint32_t acc_cols = 2u * half_cols; // of a buffer: large and small terms
  // the K steps [from, to) of 32 bytes that block chunk `c` and filter column `s` really need
  const int per_chunk = p.BK / 32;
  auto step_from = [&](int s, int c) { return s == 0 ? max(q.skip_first - per_chunk * c, 0) : 0; };
  auto step_to = [&](int s, int c) { return min(p.ksteps, (s == p.kw - 1 ? q.keep_last : 1 << 20) - per_chunk * c); };

  pdl_trigger();
  if (threadIdx.x == 0) {
    const int gave_up = *reinterpret_cast<volatile int *>(p.err); // read early, as in conv_gemm_body
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(bar_full + 8 * s, 1);
      ptx::mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < q.nb; ++b) {
      ptx::mbar_init(bar_act_full + 8 * b, 1);
      ptx::mbar_init(bar_act_empty + 8 * b, 1);
      ptx::mbar_init(bar_lo_full + 8 * b, kTransformWarps);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(bar_acc_full + 8 * b, 1);
      ptx::mbar_init(bar_acc_empty + 8 * b, kEpilogueWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *abort_flag = gave_up;
  }
  if (warp == 1) ptx::tcgen05_alloc(ptx::smem_u32(tmem_slot), (uint32_t)p.tmem_cols);
  if (q.mode == 2) {
    // the zero tails of the activation (and remainder) buffers, and the column table
    const int tail = (q.act_stride - q.act_bytes) / 16, bufs = q.nb * 2;
    for (int i = threadIdx.x; i < tail * bufs; i += blockDim.x)
      *reinterpret_cast<uint4 *>(smem + kSmemHeader + (size_t)(i / tail) * q.act_stride + q.act_bytes + (i % tail) * 16) = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int j = threadIdx.x; j < 256; j += blockDim.x) {
      const int img = j / (q.Rl * q.Pc), in_img = j - img * (q.Rl * q.Pc), y = in_img / q.Pc, x = in_img - y * q.Pc;
      pix[j] = (img < q.I && y < q.R && x < q.Cw) ? (img * p.OH + y) * p.OW + x : kNoPixel;
    }
  } else {
    for (int j = threadIdx.x; j < 256; j += blockDim.x) pix[j] = j;
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (*abort_flag != 0) total_tiles = 0;
  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB2) : "memory");
  }
  // the tile's first output pixel: image, row, column
  auto pixel_tile = [&](int tm) { return tm % q.m_tiles; };
  auto first_block = [&](int tm) { return (tm / q.m_tiles) * q.blocks / q.parts; };
  auto end_block = [&](int tm) { return (tm / q.m_tiles + 1) * q.blocks / q.parts; };
  auto tile_origin = [&](int tm, int &img, int &y0, int &x0) {
    const int per = q.tiles_y * q.tiles_x;
    const int g = tm / per, t = tm - g * per;
    img = g * q.I;
    y0 = (t / q.tiles_x) * q.R;
    x0 = (t % q.tiles_x) * q.Cw;
  };
  struct Walk { // the tiles of this CTA, as in conv_gemm_body
    int tile, tm, tn;
  };
  auto next_tile = [&](Walk &w) {
    w.tile += gridDim.x;
    w.tm += walk_dm;
    w.tn += walk_dn;
    if (w.tn >= n_tiles) {
      w.tn -= n_tiles;
      ++w.tm;
    }
  };

  if (warp == 0) {
    // ---------------------------------------------------------------- producer
    if (lane == 0) {
      bool ok = true;
      auto wait = [&](uint32_t bar, uint32_t parity) {
        if (ptx::mbar_try_wait(bar, parity) || ptx::mbar_wait_bounded(bar, parity, abort_flag, wait_rounds)) return true;
        if (!*abort_flag) report_error(p.err, kErrEmptyWait);
        *abort_flag = 1;
        return false;
      };
      // activation blocks run ahead of the weight tiles, with a cursor of their own
      Walk aw{(int)blockIdx.x, walk_m0, walk_n0};
      int ab = first_block(aw.tm), a_done = 0, a_buf = 0; // block of the cursor's tile, blocks issued, buffer
      int a_cycle = 0;                   // times the buffers have been gone through
      int a_img = 0, a_y = 0, a_x = 0, a_tap_r = 0, a_tap_s = 0, a_chunk = 0;
      auto start_block = [&]() { // (tap, chunk) of block `ab`
        const int tap = ab / p.c_chunks;
        a_chunk = ab - tap * p.c_chunks;
        a_tap_r = tap / p.kw;
        a_tap_s = tap - a_tap_r * p.kw;
      };
      start_block();
      bool a_new = true;
      auto issue_block = [&]() {
        if (aw.tile >= total_tiles) return;
        if (a_cycle > 0 && !wait(bar_act_empty + 8 * a_buf, (uint32_t)(a_cycle - 1) & 1u)) {
          ok = false;
          return;
        }
        const uint32_t dst = act0 + (uint32_t)(a_buf * q.act_stride), fb = bar_act_full + 8 * a_buf;
        ptx::mbar_expect_tx(fb, (uint32_t)q.act_bytes);
        if (q.mode == 2) {
          if (a_new) tile_origin(pixel_tile(aw.tm), a_img, a_y, a_x);
          ptx::tma_load_4d(dst, &tmA, fb, a_chunk * p.BK, a_x - p.pl, a_y - p.pt, a_img);
        } else if (q.mode == 1) {
          if (a_new) {
            const int m0 = pixel_tile(aw.tm) * 128, t = m0 / p.OW;
            a_img = t / p.OH;
            a_y = (t - a_img * p.OH) * p.sh - p.pt;
            a_x = (m0 - t * p.OW) * p.sw - p.pl;
          }
          ptx::tma_load_im2col_4d(dst, &tmA, fb, a_chunk * p.BK, a_x, a_y, a_img, (uint16_t)(a_tap_s * p.dw), (uint16_t)(a_tap_r * p.dh));
        } else {
          ptx::tma_load_2d(dst, &tmA, fb, a_chunk * p.BK, pixel_tile(aw.tm) * 128);
        }
        a_new = false;
        ++a_done;
        if (++a_buf == q.nb) {
          a_buf = 0;
          ++a_cycle;
        }
        if (++a_chunk == p.c_chunks) {
          a_chunk = 0;
          if (++a_tap_s == p.kw) {
            a_tap_s = 0;
            ++a_tap_r;
          }
        }
        if (++ab == end_block(aw.tm)) {
          a_new = true;
          next_tile(aw);
          ab = first_block(aw.tm);
          start_block();
        }
      };
      pdl_wait(); // the activations from here on
      if (taps > 1)
        for (int i = 0; i < q.nb - 1 && ok; ++i) issue_block();
      int it = 0, ps = 0;
      uint32_t pph = 0;
      // With several taps, where in a block the one nb - 1 further is sent for: its buffer is the one the previous block
      // frees, which the MMA thread leaves about when this thread is a ring's length into the block. With one tap the
      // blocks are a plain ring beside that of the weights.
      const int ahead = min(taps - 1, p.stages);
      for (Walk w{(int)blockIdx.x, walk_m0, walk_n0}; w.tile < total_tiles && ok; next_tile(w)) {
        const int n0 = w.tn * 128;
        const int b0 = first_block(w.tm), b1 = end_block(w.tm);
        int tap = b0 / p.c_chunks, chunk = b0 - tap * p.c_chunks; // mode 1 walks (tap, chunk) by blocks, mode 2 chunks by blocks and taps inside
        for (int b = b0; b < b1 && ok; ++b) {
          int s = 0;
          for (int t = 0; t < taps; ++t) {
            if (t == ahead) issue_block();
            if (!ok) break;
            const int wt = q.mode == 2 ? t : tap;
            const bool none = q.mode == 2 && step_from(s, chunk) >= step_to(s, chunk);
            if (++s == p.kw) s = 0;
            if (none) continue;
            if (it >= p.stages && !wait(bar_empty + 8 * ps, pph ^ 1u)) {
              ok = false;
              break;
            }
            const uint32_t dst = ring0 + (uint32_t)ps * w_bytes, fb = bar_full + 8 * ps;
            ptx::mbar_expect_tx(fb, w_bytes);
            ptx::tma_load_3d(dst, &tmB, fb, chunk * p.BK, wt, n0);
            ptx::tma_load_3d(dst + w_tile, &tmB2, fb, chunk * p.BK, wt, n0);
            ++it;
            if (++ps == p.stages) {
              ps = 0;
              pph ^= 1u;
            }
          }
          if (++chunk == p.c_chunks) {
            chunk = 0;
            ++tap;
          }
        }
      }
      if (!ok || *abort_flag) {
        // drain (bounded): no copy may be in flight when the CTA's shared memory is released
        for (int j = max(it - p.stages, 0); j < it; ++j)
          for (uint32_t w = 0; w < (1u << 20); ++w)
            if (ptx::mbar_try_wait(bar_full + 8 * (j % p.stages), (uint32_t)(j / p.stages) & 1u)) break;
        for (int j = max(a_done - q.nb, 0); j < a_done; ++j)
          for (uint32_t w = 0; w < (1u << 20); ++w)
            if (ptx::mbar_try_wait(bar_act_full + 8 * (j % q.nb), (uint32_t)(j / q.nb) & 1u)) break;
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      int ms = 0, t_count = 0, a_buf = 0, buf = 0;
      uint32_t mph = 0, aph = 0, acc_ph = 1; // acc_ph: parity of the accumulators' "drained" barriers

      bool ok = true;
      auto wait = [&](uint32_t bar, uint32_t parity, int code) {
        if (ptx::mbar_try_wait(bar, parity) || ptx::mbar_wait_bounded(bar, parity, abort_flag, wait_rounds)) return true;
        if (!*abort_flag) report_error(p.err, code);
        *abort_flag = 1;
        return false;
      };
      const uint64_t desc0 = make_kmajor_desc(act0, p.BK);
      const uint32_t desc_hi = (uint32_t)(desc0 >> 32);
      const uint32_t act_lo = (uint32_t)desc0, act_step = (uint32_t)q.act_stride >> 4;
      const uint32_t rem_off = (uint32_t)(q.nb * q.act_stride) >> 4; // remainder block of the same buffer
      const uint32_t ring_lo = (uint32_t)make_kmajor_desc(ring0, p.BK), w_step = w_bytes >> 4, wl_off = w_tile >> 4;
      const uint32_t px = (uint32_t)p.BK >> 4; // one pixel of a block
      const uint32_t tap_col = (uint32_t)p.dw * px, tap_row = (uint32_t)(p.dh * q.Pc) * px - (uint32_t)(p.kw - 1) * tap_col;
      for (Walk w{(int)blockIdx.x, walk_m0, walk_n0}; w.tile < total_tiles && ok; next_tile(w), ++t_count) {
        if (t_count >= q.acc_bufs) {
          if (!wait(bar_acc_empty + 8 * buf, acc_ph, kErrAccWait)) {
            ok = false;
            break;
          }
          ptx::tcgen05_fence_after();
        }
        const uint32_t d = tmem_base + (uint32_t)buf * acc_cols;
        uint32_t first = 0; // "accumulate" of the next product
        const int b0 = first_block(w.tm), b1 = end_block(w.tm);
        int chunk = q.mode == 2 ? b0 : 0; // (only tap blocks look at it)
        for (int b = b0; b < b1 && ok; ++b) {
          if (!wait(bar_lo_full + 8 * a_buf, aph, kErrFullWait)) {
            ok = false;
            break;
          }
          uint32_t x = act_lo + (uint32_t)a_buf * act_step;
          int s = 0;
          for (int t = 0; t < taps; ++t) {
            const int from = q.mode == 2 ? step_from(s, chunk) : 0, to = q.mode == 2 ? step_to(s, chunk) : p.ksteps;
            if (from < to) {
              if (!wait(bar_full + 8 * ms, mph, kErrFullWait)) {
                ok = false;
                break;
              }
              ptx::tcgen05_fence_after();
              const uint32_t wd = ring_lo + (uint32_t)ms * w_step;
              const uint32_t r = x + rem_off, wr = wd + wl_off;
              for (int k = from; k < to; ++k) {
                ptx::tcgen05_mma_tf32_lohi<false>(d + half_cols, wd + 2 * k, desc_hi, r + 2 * k, desc_hi, p.idesc, first);
                ptx::tcgen05_mma_tf32_lohi<true>(d + half_cols, wr + 2 * k, desc_hi, x + 2 * k, desc_hi, p.idesc, 1u);
                ptx::tcgen05_mma_tf32_lohi<false>(d, wd + 2 * k, desc_hi, x + 2 * k, desc_hi, p.idesc, first);
                first = 1u;
              }
              ptx::tcgen05_commit(bar_empty + 8 * ms);
              if (++ms == p.stages) {
                ms = 0;
                mph ^= 1u;
              }
            }
            x += tap_col;
            if (++s == p.kw) {
              s = 0;
              x += tap_row - tap_col;
            }
          }
          if (!ok) break;
          ptx::tcgen05_commit(bar_act_empty + 8 * a_buf);
          if (++a_buf == q.nb) {
            a_buf = 0;
            aph ^= 1u;
          }
          if (++chunk == p.c_chunks) chunk = 0;
        }
        if (ok) ptx::tcgen05_commit(bar_acc_full + 8 * buf);
        if (++buf == q.acc_bufs) {
          buf = 0;
          acc_ph ^= 1u;
        }
      }
    }
  } else if (warp < 2 + kEpilogueWarps) {
    // ---------------------------------------------------------------- epilogue
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    float bias_f = 0.0f;
    int staged_n0 = -1, buf = 0;
    uint32_t acc_ph = 0;
    bool ok = true;
    const int ch_base = p.group > 1 ? (quarter * 32) & (128 / p.group - 1) : quarter * 32;
    const size_t px_off = p.group > 1 ? (size_t)(quarter * 32 * p.group >> 7) * p.ldc_px : 0;
    pdl_wait(); // results go where an earlier kernel may still read
    for (Walk w{(int)blockIdx.x, walk_m0, walk_n0}; w.tile < total_tiles && ok; next_tile(w)) {
      const int n0 = w.tn * 128;
      const int ch = n0 + ch_base + lane;
      if (n0 != staged_n0) {
        bias_f = ch < p.n_valid ? __int_as_float(p.bias[ch]) : 0.0f;
        staged_n0 = n0;
      }
      TableMap map{pix, 0};
      size_t m0;
      if (q.mode == 2) {
        int img, y0, x0;
        tile_origin(pixel_tile(w.tm), img, y0, x0);
        m0 = ((size_t)img * p.OH + y0) * p.OW + x0;
        map.lim = q.I > 1 ? (q.images - img) * p.OH * p.OW : (p.OH - y0) * p.OW - x0;
      } else {
        m0 = (size_t)pixel_tile(w.tm) * 128;
        map.lim = p.M_total - (int)m0;
      }
      ok = ptx::mbar_wait_bounded(bar_acc_full + 8 * buf, acc_ph, abort_flag, wait_rounds);
      if (!ok && !*abort_flag) {
        report_error(p.err, kErrAccWait);
        *abort_flag = 1;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      ptx::tcgen05_fence_after();
      if (n0 + ch_base < p.n_valid) { // warp-uniform: this lane quarter holds real outputs
        const uint32_t lane_addr = tmem_base + (uint32_t)buf * acc_cols + ((uint32_t)(quarter * 32) << 16);
        constexpr int H = kEpilogueWarps / 4;
        uint8_t *out = reinterpret_cast<uint8_t *>(p.out) + m0 * p.ldc + px_off + (size_t)(w.tm / q.m_tiles) * q.part_bytes + (size_t)ch * 4;
        if (p.act == 1) epilogue_channels_f32<true>(p, lane_addr, out, ch < p.n_valid, half, H, bias_f, q.n_used, half_cols, map);
        else epilogue_channels_f32<false>(p, lane_addr, out, ch < p.n_valid, half, H, bias_f, q.n_used, half_cols, map);
      }
      ptx::tcgen05_fence_before();
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_acc_empty + 8 * buf) : "memory");
      if (++buf == q.acc_bufs) {
        buf = 0;
        acc_ph ^= 1u;
      }
    }
  } else {
    // ------------------------------------------------- remainder blocks: xl = x - (upper 19 bits of x), same layout
    const int tid = threadIdx.x - 32 * (2 + kEpilogueWarps);
    const int vecs = q.act_bytes / 16;
    int a_buf = 0;
    uint32_t aph = 0;
    bool ok = true;
    for (Walk w{(int)blockIdx.x, walk_m0, walk_n0}; w.tile < total_tiles && ok; next_tile(w))
      for (int b = first_block(w.tm), b1 = end_block(w.tm); b < b1; ++b) {
        ok = ptx::mbar_wait_bounded(bar_act_full + 8 * a_buf, aph, abort_flag, wait_rounds);
        if (!ok && !*abort_flag) {
          report_error(p.err, kErrFullWait);
          *abort_flag = 1;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint4 *src = reinterpret_cast<const uint4 *>(smem + (act0 - base) + (size_t)a_buf * q.act_stride);
        float4 *dst = reinterpret_cast<float4 *>(smem + (lo0 - base) + (size_t)a_buf * q.act_stride);
        for (int i = tid; i < vecs; i += 32 * kTransformWarps) {
          const uint4 v = src[i];
          dst[i] = make_float4(__fsub_rn(__uint_as_float(v.x), __uint_as_float(v.x & 0xffffe000u)),
                               __fsub_rn(__uint_as_float(v.y), __uint_as_float(v.y & 0xffffe000u)),
                               __fsub_rn(__uint_as_float(v.z), __uint_as_float(v.z & 0xffffe000u)),
                               __fsub_rn(__uint_as_float(v.w), __uint_as_float(v.w & 0xffffe000u)));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // visible to the tensor core
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_lo_full + 8 * a_buf) : "memory");
        if (++a_buf == q.nb) {
          a_buf = 0;
          aph ^= 1u;
        }
      }
  }

  ptx::tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tcgen05_fence_after();
    ptx::tcgen05_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
}

// Adds the parts of a TF32 launch (TapParams::parts) in order, then bias and ReLU; one 16-byte vector per thread.
__global__ void tf32_reduce_kernel(const float4 *__restrict__ ws, float4 *__restrict__ out, const float4 *__restrict__ bias, size_t nvec,
                                   int vecs_per_px, int parts, int relu) {
  pdl_prologue();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nvec; i += (size_t)gridDim.x * blockDim.x) {
    float4 s = ws[i];
    for (int k = 1; k < parts; ++k) {
      const float4 v = ws[i + (size_t)k * nvec];
      s = make_float4(__fadd_rn(s.x, v.x), __fadd_rn(s.y, v.y), __fadd_rn(s.z, v.z), __fadd_rn(s.w, v.w));
    }
    const float4 b = bias[i % vecs_per_px];
    s = make_float4(__fadd_rn(s.x, b.x), __fadd_rn(s.y, b.y), __fadd_rn(s.z, b.z), __fadd_rn(s.w, b.w));
    if (relu) s = make_float4(s.x > 0.f ? s.x : 0.f, s.y > 0.f ? s.y : 0.f, s.z > 0.f ? s.z : 0.f, s.w > 0.f ? s.w : 0.f);
    out[i] = s;
  }
}

} // namespace tpucb
