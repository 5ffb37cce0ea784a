// The implicit-GEMM convolution of conv_gemm_i8.cuh for launches that fill the GPU: one CTA per SM with up to 256 pixels per
// tile, and for layers of many channels a pair of CTAs (two SMs) per tile.
//
// What bounds the tiles of 128 channels x 128 pixels there is shared memory: 122 to 125 of the 128 bytes that an SM's serves
// per clock, half for the tensor core's operands, half for the copies that bring them (res4 3x3 layer of ResNet-50, batch 256,
// 1.70 POP/s). Here
//   pair (CTAS = 2, tcgen05 cta_group::2): 256 channels x NT pixels, each CTA holding the weights of its 128 channels and half
//     of the pixels; the tensor cores read the other half from the other SM. For NT = 256 that is half the bytes per
//     multiply-add on both sides;
//   single (CTAS = 1): 128 channels x NT pixels, three quarters of the operand reads and of the copies for NT = 256.
// The epilogue is bound by instruction issue in layers with a short K. It reads the accumulators in the fragment layout of the
// matrix stores (tcgen05.ld.16x256b: a lane holds two channels x two pixels), so that stmatrix leaves whole pixels in shared
// memory, and one bulk tensor store per 32 pixels x 128 bytes writes them, clipped to the tensor by its map: no lane
// computes an address or a bound.
//
// Warps (608 threads): 0 copies activations, 1 copies weights, 2 owns tensor memory and issues the MMAs (of the pair: in its
// first CTA), 3..18 are the epilogue: four groups of four, a group taking every fourth column group of 32 pixels. Every wait
// is bounded as there: on expiry the CTA records an error code, its roles fall through to the common end.
#pragma once
#include "conv_gemm_i8.cuh"

namespace tpucb {

constexpr int kBigEpilogueWarps = 16;
constexpr int kBigThreads = 32 * (3 + kBigEpilogueWarps);
constexpr int kBigHeader = 1024; // barriers
// staging of the results: per epilogue group 32 pixels x 128 channels, twice for one-byte values
constexpr int kBigStaging[3] = {4 * 2 * 4096, 4 * 8192, 4 * 16384};

namespace ptx {
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of `addr` (own shared memory) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_cluster(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
template <int CTAS> __device__ __forceinline__ void big_load_2d(uint32_t dst, const void *tmap, uint32_t bar, int x, int y) {
  if constexpr (CTAS == 1) tma_load_2d(dst, tmap, bar, x, y);
  else
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%3, %4}], [%2];" ::"r"(dst), "l"(tmap), "r"(bar), "r"(x), "r"(y) : "memory");
}
template <int CTAS> __device__ __forceinline__ void big_load_3d(uint32_t dst, const void *tmap, uint32_t bar, int x, int y, int z) {
  if constexpr (CTAS == 1) tma_load_3d(dst, tmap, bar, x, y, z);
  else
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst), "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
template <int CTAS>
__device__ __forceinline__ void big_load_im2col(uint32_t dst, const void *tmap, uint32_t bar, int c, int w, int h, int n, uint16_t off_w,
                                                uint16_t off_h) {
  if constexpr (CTAS == 1) tma_load_im2col_4d(dst, tmap, bar, c, w, h, n, off_w, off_h);
  else
    asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.im2col.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};" ::"r"(dst), "l"(tmap), "r"(bar), "r"(c), "r"(w), "r"(h), "r"(n),
                 "h"(off_w), "h"(off_h) : "memory");
}
__device__ __forceinline__ void tma_store_2d(const void *tmap, uint32_t src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(tmap), "r"(src), "r"(x), "r"(y)
               : "memory");
}
// arrives on the barrier at this offset in every CTA of the tile when the MMAs issued so far have been done
template <int CTAS> __device__ __forceinline__ void big_commit(uint32_t bar) {
  if constexpr (CTAS == 1) tcgen05_commit(bar);
  else
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3) : "memory");
}
template <int CTAS, int KIND>
__device__ __forceinline__ void big_mma(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
#define TPUCB_MMA(GROUP, K)                                                                                                          \
  asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\tsetp.ne.b32 p, %5, 0;\n\t" \
               "tcgen05.mma." GROUP ".kind::" K " [%0], da, db, %4, p;\n\t}" ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc),      \
               "r"(accumulate) : "memory")
  if constexpr (CTAS == 1) {
    if (KIND == 0) TPUCB_MMA("cta_group::1", "i8");
    else if (KIND == 1) TPUCB_MMA("cta_group::1", "f16");
    else TPUCB_MMA("cta_group::1", "tf32");
  } else {
    if (KIND == 0) TPUCB_MMA("cta_group::2", "i8");
    else if (KIND == 1) TPUCB_MMA("cta_group::2", "f16");
    else TPUCB_MMA("cta_group::2", "tf32");
  }
#undef TPUCB_MMA
}
// 16 lanes x 32 columns: r[4 i + ...] = (lane t/4, column 8 i + 2 (t % 4)), (same, + 1), (lane t/4 + 8, ...), (same, + 1)
__device__ __forceinline__ void tcgen05_ld_frag(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ void stmatrix_b8(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m16n8.x4.trans.shared.b8 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void stmatrix_b16(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
} // namespace ptx

// FORM (INT8): of the requantisation, 1 requant_fast, 3 float_requant2. ACT: 0 none, 1 ReLU, 2 leaky.
template <int CTAS, int KIND, int ACT, int FORM>
__device__ __forceinline__ void conv_big_body(const CUtensorMap &tmA, const CUtensorMap &tmB, const CUtensorMap &tmA2,
                                              const CUtensorMap &tmB2, const CUtensorMap &tmO, const CUtensorMap &tmO2,
                                              const ConvGemmParams &p) {
  constexpr bool TF32 = KIND == 2;
  constexpr int kTerms = TF32 ? 3 : 1;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (base - raw);
  const uint32_t bar_full = base, bar_empty = base + 64, bar_acc_full = base + 128, bar_acc_empty = base + 144;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 168);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 172);

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = CTAS == 1 ? 0u : ptx::cluster_rank();
  const int nt = p.m_tile; // pixels per tile
  const int px_cta = nt / CTAS;
  const int n_tiles = (p.n_valid + 128 * CTAS - 1) / (128 * CTAS), m_tiles = (p.M_total + nt - 1) / nt;
  int total = n_tiles * m_tiles;
  const int first = (int)blockIdx.x / CTAS, step = (int)gridDim.x / CTAS;
  const uint32_t a_bytes = (uint32_t)px_cta * (uint32_t)p.BK, b_bytes = 128u * (uint32_t)p.BK;
  const uint32_t stage_bytes = a_bytes + b_bytes;
  const uint32_t staging = base + kBigHeader, ring = staging + kBigStaging[KIND];
  const int taps = p.kh * p.kw, k_iters = taps * p.c_chunks;
  const int wait_rounds = p.wait_rounds > 0 ? p.wait_rounds : 1024;

  pdl_trigger();
  if (threadIdx.x == 0) {
    const int gave_up = *reinterpret_cast<volatile int *>(p.err); // as in conv_gemm_body
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(bar_full + 8 * s, 2); // one arrival per copying warp, with the bytes of all CTAs of the tile
      ptx::mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(bar_acc_full + 8 * b, 1);
      ptx::mbar_init(bar_acc_empty + 8 * b, CTAS * kBigEpilogueWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *abort_flag = gave_up;
  }
  if (warp == 2) {
    if constexpr (CTAS == 1) {
      ptx::tcgen05_alloc(ptx::smem_u32(tmem_slot), 512u);
    } else {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(ptx::smem_u32(tmem_slot)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  if constexpr (CTAS > 1) ptx::cluster_sync(); // the other CTA's barriers are ready as well
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  if (*abort_flag != 0) {
    if constexpr (CTAS == 1) total = 0;
    // (A pair goes on: one CTA may have seen the flag and the other not. Its waits are bounded.)
  }
  // barriers of the pair's first CTA, which counts the copies of both and issues the MMAs
  const uint32_t lead_full = CTAS == 1 ? bar_full : ptx::map_cluster(bar_full, 0);

  if (warp <= 1) {
    // ------------------------------------------------------------ copies: warp 0 the activations, warp 1 the weights
    {
      const bool acts = warp == 0;
      if (ptx::elect_one()) asm volatile("prefetch.tensormap [%0];" ::"l"(acts ? &tmA : &tmB) : "memory");
      if (acts) pdl_wait(); // weights are written at load time only: their copies need not wait for the previous kernel
      const uint32_t bytes = acts ? a_bytes : b_bytes, dst0 = ring + (acts ? 0u : a_bytes);
      int it = 0, ps = 0;
      uint32_t pph = 0;
      bool ok = true;
      for (int tile = first; tile < total && ok; tile += step) {
        const int tm = tile / n_tiles, tn = tile - tm * n_tiles;
        const int n0 = (tn * CTAS + (int)rank) * 128;
        int m0 = tm * nt + (int)rank * px_cta;
        if (m0 >= p.M_total) m0 = 0; // the second half of the last tile: any pixels, nothing of them is written
        int n_img = 0, h_base = 0, w_base = 0;
        if (acts && p.a_mode == 1) {
          const int q = m0 % p.OW, t = m0 / p.OW, pp = t % p.OH;
          n_img = t / p.OH;
          w_base = q * p.sw - p.pl;
          h_base = pp * p.sh - p.pt;
        }
        int tap = 0, tr = 0, ts = 0, chunk = 0, term = 0;
        for (int kit = 0; kit < kTerms * k_iters; ++kit, ++it) {
          if (it >= p.stages && !ptx::mbar_wait_warp(bar_empty + 8 * ps, pph ^ 1u, abort_flag, wait_rounds)) {
            wait_expired(p.err, abort_flag, kErrEmptyWait);
            ok = false;
            break;
          }
          const uint32_t dst = dst0 + (uint32_t)ps * stage_bytes;
          const int c0 = chunk * p.BK;
          const uint32_t fb = lead_full + 8 * ps;
          if (ptx::elect_one()) {
            if (rank == 0) ptx::mbar_expect_tx(bar_full + 8 * ps, CTAS * bytes);
            if (!acts) ptx::big_load_3d<CTAS>(dst, (TF32 && term == 1) ? &tmB2 : &tmB, fb, c0, tap, n0);
            else if (p.a_mode == 1)
              ptx::big_load_im2col<CTAS>(dst, (TF32 && term == 0) ? &tmA2 : &tmA, fb, c0, w_base, h_base, n_img, (uint16_t)(ts * p.dw),
                                         (uint16_t)(tr * p.dh));
            else ptx::big_load_2d<CTAS>(dst, (TF32 && term == 0) ? &tmA2 : &tmA, fb, c0, m0);
          }
          if (++chunk == p.c_chunks) {
            chunk = 0;
            ++tap;
            if (++ts == p.kw) {
              ts = 0;
              ++tr;
            }
            if (TF32 && tap == taps) {
              tap = tr = ts = 0;
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
        // No copy may be in flight when the CTA's shared memory is released, and the barriers that would tell may count
        // copies that were never started: a copy lands within microseconds, so 2 ms are waited for, by the clock.
        unsigned long long t0, t1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        for (int i = 0; i < (1 << 20); ++i) {
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
          if (t1 - t0 > 2000000ull) break;
          __nanosleep(1000);
        }
      }
    }
  } else if (warp == 2) {
    // ---------------------------------------------------------------------------------------------------- MMA issuer
    if (rank == 0) {
      int t = 0, ms = 0;
      uint32_t mph = 0;
      bool ok = true;
      const uint64_t desc0 = make_kmajor_desc(ring, p.BK);
      const uint32_t hi = (uint32_t)(desc0 >> 32), ring_lo0 = (uint32_t)desc0;
      const uint32_t stage_step = stage_bytes >> 4, w_at = a_bytes >> 4;
      uint32_t m_full = bar_full, m_empty = bar_empty, lo = ring_lo0;
      const int ksteps = p.ksteps;
      for (int tile = first; tile < total && ok; tile += step, ++t) {
        const int buf = t & 1;
        if (t >= 2) {
          if (!ptx::mbar_wait_warp(bar_acc_empty + 8 * buf, (uint32_t)(((t >> 1) - 1) & 1), abort_flag, wait_rounds)) {
            wait_expired(p.err, abort_flag, kErrAccWait);
            break;
          }
          ptx::tcgen05_fence_after();
        }
        const uint32_t d = tmem_base + (uint32_t)buf * 256u;
        // (two copies of the loop, as in conv_gemm_body: whole K blocks, and those with a padded tail)
        auto k_loop = [&](auto whole) {
          for (int kit = 0; kit < kTerms * k_iters; ++kit) {
            if (!ptx::mbar_wait_warp(m_full, mph, abort_flag, wait_rounds)) {
              wait_expired(p.err, abort_flag, kErrFullWait);
              ok = false;
              break;
            }
            ptx::tcgen05_fence_after();
            const uint32_t w_lo = lo + w_at;
            if (ptx::elect_one()) {
              if constexpr (decltype(whole)::value) {
                ptx::big_mma<CTAS, KIND>(d, w_lo, lo, hi, p.idesc, kit > 0 ? 1u : 0u);
#pragma unroll
                for (int k = 1; k < 4; ++k) ptx::big_mma<CTAS, KIND>(d, w_lo + 2 * k, lo + 2 * k, hi, p.idesc, 1u);
              } else {
                for (int k = 0; k < ksteps; ++k) ptx::big_mma<CTAS, KIND>(d, w_lo + 2 * k, lo + 2 * k, hi, p.idesc, kit + k > 0 ? 1u : 0u);
              }
              ptx::big_commit<CTAS>(m_empty);
            }
            m_full += 8;
            m_empty += 8;
            lo += stage_step;
            if (++ms == p.stages) {
              ms = 0;
              mph ^= 1u;
              m_full = bar_full;
              m_empty = bar_empty;
              lo = ring_lo0;
            }
          }
        };
        if (ksteps == 4) k_loop(std::true_type{});
        else k_loop(std::false_type{});
        if (ok && ptx::elect_one()) ptx::big_commit<CTAS>(bar_acc_full + 8 * buf);
      }
    }
  } else {
    // ------------------------------------------------------------------------------------------------------ epilogue
    const int quarter = warp & 3, group = (warp - 3) >> 2;
    const bool issuer = (warp - 3) % 4 == 0 && lane == 0; // starts the group's stores
    const uint32_t stage = staging + (uint32_t)group * (kBigStaging[KIND] / 4);
    const uint32_t lead_acc_empty = CTAS == 1 ? bar_acc_empty : ptx::map_cluster(bar_acc_empty, 0);
    const int row_xor = (lane & 7) << 4; // the 128-byte swizzle of pixel `lane` of a block of 32
    const uint32_t stage_row = (uint32_t)lane * 128u;
    FloatRequantPairs<ACT == 1> fq[4];
    FloatRequantShared fshared = {};
    if constexpr (FORM == 3 && ACT != 1) fshared.set();
    ChanConst cc[4];
    float bias[4];
    unsigned long long bias2[4];
    int staged_n0 = -1, t = 0, flip = 0;
    auto sync_group = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); };
    pdl_wait();
    for (int tile = first; tile < total; tile += step, ++t) {
      const int tm = tile / n_tiles, tn = tile - tm * n_tiles;
      const int m0 = tm * nt, n0 = (tn * CTAS + (int)rank) * 128, buf = t & 1;
      if (n0 != staged_n0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int ch = n0 + quarter * 32 + (TF32 ? lane : (lane >> 2) + 8 * i);
          const bool v = ch < p.n_valid;
          if (KIND != 0) {
            bias[i] = v ? __int_as_float(__ldg(p.bias + ch)) : 0.0f;
            if (KIND == 1) bias2[i] = hold_pair(bias[i]);
          } else if (FORM == 3) {
            const uint4 c = v ? __ldg(reinterpret_cast<const uint4 *>(p.fq) + ch) : make_uint4(0u, 0u, 0u, 0u);
            fq[i].set(FloatRequant{c.x, __uint_as_float(c.y), __uint_as_float(c.z), __uint_as_float(c.w)});
          } else {
            cc[i] = load_chan_const(p, ch);
          }
        }
        staged_n0 = n0;
      }
      bool ok = *abort_flag == 0;
      if (ok) ok = ptx::mbar_wait_bounded(bar_acc_full + 8 * buf, (uint32_t)((t >> 1) & 1), abort_flag, wait_rounds);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) wait_expired(p.err, abort_flag, kErrAccWait);
      // After an expired wait a warp does no more work, but it comes to every barrier of its group.
      ptx::tcgen05_fence_after();
      const int cols = min(nt, p.M_total - m0); // this tile's pixels
      const bool mine = ok && n0 + quarter * 32 < p.n_valid;
      const int last = group * 32 + ((cols - 1 - group * 32) & ~127); // this group's last column group of the tile
      const uint32_t acc = tmem_base + (uint32_t)buf * 256u + ((uint32_t)(quarter * 32) << 16);
      auto release = [&]() { // the accumulator buffer goes back to the MMA issuer
        ptx::tcgen05_fence_before();
        __syncwarp();
        if (lane == 0 && !p.lose_arrival) {
          if constexpr (CTAS == 1) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_acc_empty + 8 * buf) : "memory");
          else asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(lead_acc_empty + 8 * buf) : "memory");
        }
      };
      if (group * 32 >= cols) release();
      for (int col = group * 32; col < cols; col += 128) {
        uint32_t w[KIND == 0 ? 8 : 16];
        uint32_t r0[16], r1[16];
        if (mine) {
          if constexpr (TF32) {
            ptx::tcgen05_ld_x16(acc + (uint32_t)col, r0);
            ptx::tcgen05_ld_x16(acc + (uint32_t)col + 16u, r1);
          } else {
            ptx::tcgen05_ld_frag(acc + (uint32_t)col, r0);
            ptx::tcgen05_ld_frag(acc + (uint32_t)col + (16u << 16), r1);
          }
          ptx::tcgen05_wait_ld();
        }
        if (col == last) release();
        if constexpr (KIND == 0) {
          if (mine) {
            // word k of half h: channels t/4 and t/4 + 8 of the half's sixteen, pixels 8 k + 2 (t % 4) and + 1
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const int h = k >> 2;
              const uint32_t *r = h ? r1 + 4 * (k & 3) : r0 + 4 * (k & 3);
              int v[4];
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                const int c = 2 * h + j;
                if constexpr (FORM == 3) {
                  float_requant2<ACT == 1>(r[2 * j], r[2 * j + 1], fq[c], fshared, v[2 * j], v[2 * j + 1]);
                } else {
                  v[2 * j] = requant_fast<ACT == 1 ? 1 : 0, false>((int32_t)r[2 * j], cc[c], p);
                  v[2 * j + 1] = requant_fast<ACT == 1 ? 1 : 0, false>((int32_t)r[2 * j + 1], cc[c], p);
                }
              }
              if constexpr (FORM == 3) w[k] = float_requant_pack<ACT == 1>(v[0], v[1], v[2], v[3]);
              else w[k] = ACT == 1 ? relu_bytes(pack4_sat(v[0], v[1], v[2], v[3])) : pack4_sat(v[0], v[1], v[2], v[3]);
            }
          }
          // Two buffers per group: the issuer waits for the store before the last one's reads ahead of the barrier, so that
          // past it that store's buffer is free.
          auto send = [&](const CUtensorMap *map) {
            if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
            const uint32_t at = stage + (uint32_t)flip * 4096u;
            if (mine) {
#pragma unroll
              for (int h = 0; h < 2; ++h)
                ptx::stmatrix_b8(at + stage_row + (uint32_t)(((quarter * 2 + h) << 4) ^ row_xor), w[4 * h], w[4 * h + 1], w[4 * h + 2],
                                 w[4 * h + 3]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            sync_group();
            if (issuer && ok && n0 < p.n_valid) {
              ptx::tma_store_2d(map, at, n0, m0 + col);
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            flip ^= 1;
          };
          if (ACT != 2 || p.out2) send(&tmO);
          if (ACT == 2) { // leaky ReLU on the packed, saturated values
#pragma unroll
            for (int k = 0; k < 8; ++k) w[k] = leaky4(w[k], p);
            send(&tmO2);
          }
        } else {
          // One buffer per group: it is free once the issuer has waited for the last store's reads and the group has met.
          if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
          if constexpr (KIND == 1) {
            if (mine) {
              uint32_t odd = 0u;
              // word j of half h: (channel t/4, two pixels), (channel t/4 + 8, two pixels), ...
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const uint32_t x0 = j < 8 ? r0[2 * j] : r1[2 * j - 16], x1 = j < 8 ? r0[2 * j + 1] : r1[2 * j - 15];
                unsigned long long v = pack_b32x2(x0, x1);
                asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(bias2[2 * (j >> 3) + (j & 1)]));
                w[j] = bf16_pack_relu<ACT == 1>(v, odd);
              }
              if (odd & 0x7fff7fffu) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                  const uint32_t x0 = j < 8 ? r0[2 * j] : r1[2 * j - 16], x1 = j < 8 ? r0[2 * j + 1] : r1[2 * j - 15];
                  w[j] = bf16_pack_rule<ACT == 1>(x0, x1, __uint_as_float((uint32_t)bias2[2 * (j >> 3) + (j & 1)]));
                }
              }
            }
            sync_group();
            if (mine) {
              // sixteen-byte column 4 quarter + 2 h + i of the pixel's 256: 64 channels per store
#pragma unroll
              for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                  const int c16 = quarter * 4 + 2 * h + i;
                  ptx::stmatrix_b16(stage + (uint32_t)(c16 >> 3) * 4096u + stage_row + (uint32_t)(((c16 & 7) << 4) ^ row_xor), w[8 * h + i],
                                    w[8 * h + i + 2], w[8 * h + i + 4], w[8 * h + i + 6]);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            sync_group();
            if (issuer && ok) {
              for (int i = 0; i < 2; ++i)
                if (n0 + 64 * i < p.n_valid) ptx::tma_store_2d(&tmO, stage + 4096u * i, 2 * (n0 + 64 * i), m0 + col);
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
          } else {
            // fp32: a lane owns a channel, a warp's 32 channels are 128 bytes of a pixel and a store of their own
            sync_group();
            const uint32_t at = stage + (uint32_t)quarter * 4096u + (uint32_t)lane * 4u;
            auto put = [&](bool remainder) {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                float v = __fadd_rn(bits_f32(j < 16 ? r0[j & 15] : r1[j & 15]), bias[0]);
                if (ACT == 1) v = v > 0.0f ? v : 0.0f;
                if (remainder) v = __fsub_rn(v, __uint_as_float(__float_as_uint(v) & 0xffffe000u));
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + 128u * j), "f"(v) : "memory");
              }
            };
            auto send = [&](const CUtensorMap *map) {
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
              sync_group();
              if (issuer && ok) {
                for (int i = 0; i < 4; ++i)
                  if (n0 + 32 * i < p.n_valid) ptx::tma_store_2d(map, stage + 4096u * i, 4 * (n0 + 32 * i), m0 + col);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
              }
            };
            if (mine) put(false);
            send(&tmO);
            if (p.out2) { // the remainder operand of a TF32 x 3 convolution that reads this result
              if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
              __syncwarp();
              sync_group();
              if (mine) put(true);
              send(&tmO2);
            }
          }
        }
      }
    }
    if (issuer) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  ptx::tcgen05_fence_before();
  __syncthreads();
  if constexpr (CTAS > 1) ptx::cluster_sync(); // no CTA leaves while the other's arrivals or operand reads may come to it
  if (warp == 2) {
    ptx::tcgen05_fence_after();
    if constexpr (CTAS == 1) ptx::tcgen05_dealloc(tmem_base, 512u);
    else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

template <int CTAS, int KIND, int ACT, int FORM>
__global__ void __launch_bounds__(kBigThreads, 1) __cluster_dims__(CTAS, 1, 1)
conv_big_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmO,
                const __grid_constant__ CUtensorMap tmO2, const ConvGemmParams p) {
  conv_big_body<CTAS, KIND, ACT, FORM>(tmA, tmB, tmA, tmB, tmO, tmO2, p);
}
template <int CTAS, int ACT>
__global__ void __launch_bounds__(kBigThreads, 1) __cluster_dims__(CTAS, 1, 1)
conv_big_tf32x3_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmA2,
                       const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ CUtensorMap tmO,
                       const __grid_constant__ CUtensorMap tmO2, const ConvGemmParams p) {
  conv_big_body<CTAS, 2, ACT, 0>(tmA, tmB, tmA2, tmB2, tmO, tmO2, p);
}

} // namespace tpucb
