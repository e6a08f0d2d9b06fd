// The panel GEMM on narrow tiles (128 x BN, BN = 32, 64 or 128), one SM per tile, for calls whose 256-wide tiles are
// too few to fill the GPU.
//
// Same panels, products, order and promotion interval as tcec_gemm_panels.cuh, so the same bits as long as K is not divided
// (kSplit = false).  With 64 x 4096 x 4096 the wide kernel has 16 tiles for 148 SMs, this one 128.
//
// kSplit: the CTAs of a cluster share one tile and divide its K.  Every CTA walks its part like a tile of that length; the
// results, main and correction folded, are added in the order of K through the cluster's shared memory, each CTA adding and storing
// its share of the tile's warp blocks.  Fewer and wider tiles then fill the GPU, and what an SM takes in, which is what
// bounds this kernel, shrinks: a K block of a 128 x 128 tile is 32 KB for four times the products of a 128 x 32 one's 20 KB.  The
// correction, which the tensor core accumulates with truncation, covers only a part of K, so the error is no larger; the bits are
// others than those of the undivided kernels.
//
// What bounds it: the copies.  A K block of a 128 x 32 tile brings 16 + 4 KB for 240 tensor cycles (an MMA with N = 32
// takes 40 cycles, 64: 48, 128: 64), which is more than an SM takes in at 64 bytes per cycle; rows of A's panel that lie
// beyond the matrix are therefore not copied (64 rows of A: 8 + 4 KB).  Up to 200 KB of copies are in flight.
// Both accumulators exist twice in TMEM, so promotions, which a tile of long K has many of, cost no tensor time.
#pragma once
#include "tcec_gemm_panels.cuh"
#include "tcec_gemm_roles.cuh"

namespace tcec_sm100 {

template <int BN, bool kEc, bool kSplit = false>
struct GemmNarrowCfg {
  static constexpr int NP = kEc ? 2 : 1;
  static constexpr int KBS = BN == 128 ? 1 : 2;          // K blocks per stage
  static constexpr int A_BLOCK = kPanelBytes * NP;        // hi (lo) of 128 rows
  static constexpr int B_IMAGE = BN * 64;                 // hi or lo of BN rows
  static constexpr int B_BLOCK = B_IMAGE * NP;
  static constexpr int STAGE_BYTES = KBS * (A_BLOCK + B_BLOCK);
  static constexpr int EPI_WARPS = BN == 32 ? 4 : 8;
  static constexpr int NC = BN == 128 ? 64 : 32;          // columns per epilogue warp
  static constexpr int PART_BYTES = 32 * NC * 4;          // divided K: what one CTA adds to one warp block
  static constexpr int PARTS_BYTES = kSplit ? EPI_WARPS * PART_BYTES : 0;
  static constexpr int NST_RAW = (200 * 1024 - PARTS_BYTES) / STAGE_BYTES;
  static constexpr int NST = NST_RAW > 8 ? 8 : NST_RAW;
  static constexpr int PARTS_OFFSET = NST * STAGE_BYTES;
  static constexpr int EPI_OFFSET = PARTS_OFFSET + PARTS_BYTES;
  static constexpr int SMEM_BYTES = EPI_OFFSET + EPI_WARPS * kEpiBufBytes + 1024;
  static_assert(SMEM_BYTES <= 232448 - 512, "dynamic + static shared memory exceed an SM");
  static constexpr int THREADS = 128 + 32 * EPI_WARPS;
  static constexpr int TMEM_COLS = kEc ? 512 : 256;
  static constexpr int GROUP_M = 16;
};

// Stores one epilogue warp's 32 x NC block of a tile.
template <class Cfg>
__device__ __forceinline__ void store_narrow_block(const float (&acc)[Cfg::NC], const GemmPanelParams& p, const TileCoord& tc, int bn,
                                                   int q, int col_in, uint8_t* smem_gen, int ew, int lane) {
  StoreTarget st;
  st.cbase = p.c_array ? p.c_array[tc.b] : p.c + tc.b * p.c_batch_stride;
  st.ldc = p.ldc;
  st.M = p.M;
  st.N = p.N;
  st.col_major = p.c_col_major;
  st.vec_ok = !p.c_col_major && (p.ldc % 4 == 0) && ((reinterpret_cast<uintptr_t>(st.cbase) & 15) == 0);
  st.alpha = p.alpha;
  st.beta = p.beta;
  const int row0 = tc.mt * 128 + q * 32, col0 = tc.nt * bn + col_in;
  if (row0 < p.M && col0 < p.N)
    store_warp_block<true>(acc, row0, col0, st, reinterpret_cast<float*>(smem_gen + Cfg::EPI_OFFSET) + ew * kEpiBufFloats, lane);
}

// Divided K: launched with clusters of 2, 4 or 8 CTAs, one cluster per tile.
template <int BN, bool kTf32, bool kEc, bool kSplit>
__global__ void __launch_bounds__(GemmNarrowCfg<BN, kEc>::THREADS, 1) tcec_gemm_panels_narrow_kernel(const GemmPanelParams p) {
  using Cfg = GemmNarrowCfg<BN, kEc, kSplit>;
  constexpr int NST = Cfg::NST;
  if (p.only_if) {
    wait_for_launch_before();
    if (*p.only_if == 0) return;
  }
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[NST], bar_empty[NST];
  __shared__ uint64_t bar_main_full[2], bar_main_free[2], bar_corr_full[2], bar_corr_free[2], bar_drain[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ uint32_t abort_flag;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* const smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int ntiles = p.tiles_m * p.tiles_n * p.batch;
  // this CTA's tiles, and its part of their K in whole stages
  const int parts = kSplit ? static_cast<int>(cluster_nctarank()) : 1, part = kSplit ? static_cast<int>(cluster_ctarank()) : 0;
  const int first_tile = blockIdx.x / parts, stride = gridDim.x / parts;
  const int stages = (p.nkb + Cfg::KBS - 1) / Cfg::KBS;
  const int kb_first = kSplit ? stages * part / parts * Cfg::KBS : 0;
  const int kb_end = kSplit ? min(p.nkb, stages * (part + 1) / parts * Cfg::KBS) : p.nkb;
  const int nkb = kb_end - kb_first;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), kEc ? 2 : 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&bar_main_full[i]), 1);
      mbar_init(smem_u32(&bar_main_free[i]), Cfg::EPI_WARPS);
      mbar_init(smem_u32(&bar_corr_full[i]), 1);
      mbar_init(smem_u32(&bar_corr_free[i]), Cfg::EPI_WARPS);
      mbar_init(smem_u32(&bar_drain[i]), 1);
    }
    abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_s), Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (kSplit) cluster_sync_all();  // the others' shared memory exists before anything is written to it
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;  // main buffers at +0 and +128, correction buffers at +256 and +384
  volatile uint32_t* abortp = &abort_flag;
  wait_for_launch_before();

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (elect_one()) {
      uint32_t s = 0, ph = 0, armed = 0, armed_parity = 0;
      [[maybe_unused]] uint32_t it = 0;
      bool ok = true;
      auto next_stage = [&]() {
        ++it;
        if (++s == static_cast<uint32_t>(NST)) {
          s = 0;
          ph ^= 1;
        }
      };
      for (int tile = first_tile; tile < ntiles && ok; tile += stride) {
        const TileCoord tc = decode_tile(tile, p.tiles_m, p.tiles_n, Cfg::GROUP_M);
        const uint8_t* pa = p.panels_a + tc.b * p.panels_a_batch_stride + static_cast<size_t>(tc.mt) * p.nkb * Cfg::A_BLOCK;
        const int brow = tc.nt * BN;
        const uint8_t* pb = p.panels_b + tc.b * p.panels_b_batch_stride +
                            static_cast<size_t>(brow / 128) * p.nkb * (kPanelBytes * Cfg::NP) + (brow % 128) * 64;
        const int rows = (min(128, p.M - tc.mt * 128) + 7) & ~7;  // of A's panel that the matrix has, in whole groups
        for (int kb = kb_first; kb < kb_end; kb += Cfg::KBS) {
          if (!mbar_wait(smem_u32(&bar_empty[s]), ph ^ 1, abortp, 32)) {
            ok = false;
            break;
          }
          // injected stall (failure-path test): the first stage after the first ring fill is never filled, of a cluster's CTAs in one
          if (dev_flag(p.debug_flags, 64) && it == static_cast<uint32_t>(NST) && part == parts / 2) {
            next_stage();
            continue;
          }
          const uint32_t full = smem_u32(&bar_full[s]);
          const uint32_t dst = smem_base + s * Cfg::STAGE_BYTES;
          const int nblk = Cfg::KBS == 1 ? 1 : min(Cfg::KBS, kb_end - kb);
          mbar_arrive_expect_tx(full, nblk * Cfg::NP * (rows * 64 + Cfg::B_IMAGE));
          armed |= 1u << s;
          armed_parity = (armed_parity & ~(1u << s)) | (ph << s);
          const uint8_t* sa = pa + static_cast<size_t>(kb) * Cfg::A_BLOCK;
          if (rows == 128) {
            bulk_load(dst, sa, nblk * Cfg::A_BLOCK, full);
          } else {
            for (int i = 0; i < nblk * Cfg::NP; ++i) bulk_load(dst + i * kPanelBytes, sa + i * kPanelBytes, rows * 64, full);
          }
          const uint8_t* sb = pb + static_cast<size_t>(kb) * (kPanelBytes * Cfg::NP);
          const uint32_t db = dst + Cfg::KBS * Cfg::A_BLOCK;
          for (int i = 0; i < nblk * Cfg::NP; ++i) bulk_load(db + i * Cfg::B_IMAGE, sb + i * kPanelBytes, Cfg::B_IMAGE, full);
          next_stage();
        }
      }
      if (!ok) {
        abort_flag = 1;
        atomicCAS(p.status, 0, kErrProducerWait);
        // let this thread's own copies land before the CTA gives up its shared memory
        for (uint32_t q = 0; q < static_cast<uint32_t>(NST); ++q)
          if (armed & (1u << q)) mbar_wait_plain(smem_u32(&bar_full[q]), (armed_parity >> q) & 1);
      }
    }
  } else if (warp == 1 || warp == 2) {
    // ------------------------------------------------------------ MMA issuers (tcec_gemm_roles.cuh)
    if ((warp == 1 || kEc) && elect_one()) {
      DoubleImage im;
      im.dconst = umma_desc_kmajor_noswizzle(0, 128, 512);
      im.base16 = (smem_base & 0x3ffff) >> 4;
      im.stage16 = Cfg::STAGE_BYTES >> 4;
      im.a_lo16 = kPanelBytes >> 4;
      im.b_hi16 = (Cfg::KBS * Cfg::A_BLOCK) >> 4;
      im.b_lo16 = im.b_hi16 + (Cfg::B_IMAGE >> 4);
      im.kstep16 = 16;
      im.a_block16 = Cfg::A_BLOCK >> 4;
      im.b_block16 = Cfg::B_BLOCK >> 4;
      int tile = first_tile - stride;
      auto next_tile = [&](uint32_t& idesc) {
        tile += stride;
        idesc = umma_idesc(kTf32 ? 2u : 0u, 128, BN);
        return tile < ntiles;
      };
      const KWalk walk{nkb, p.promo};
      const RingBarriers ring{bar_full, bar_empty};
      const bool ok =
          warp == 1 ? issue_main_double<kTf32, NST, Cfg::KBS>(next_tile, walk, im, tmem, ring, bar_main_full, bar_main_free, abortp)
                    : issue_corr_double<kTf32, NST, Cfg::KBS>(next_tile, walk, im, tmem + 256, ring, bar_corr_full,
                                                              bar_corr_free, abortp);
      if (!ok) mma_thread_gave_up<false>(&abort_flag, p.status, kErrMmaWait, &bar_drain[warp - 1]);
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------ epilogue
    const int ew = warp - 4, q = warp & 3, col_in = (ew >> 2) * Cfg::NC;
    const uint32_t taddr = tmem + (static_cast<uint32_t>(q * 32) << 16) + col_in;
    const int nchunks = p.promo ? (nkb + p.promo - 1) / p.promo : 1;
    uint32_t chunk = 0, tcount = 0;
    bool ok = true;
    for (int tile = first_tile; tile < ntiles && ok; tile += stride, ++tcount) {
      const TileCoord tc = decode_tile(tile, p.tiles_m, p.tiles_n, Cfg::GROUP_M);
      float acc[Cfg::NC];
      for (int c = 0; c < nchunks; ++c, ++chunk) {
        if (!mbar_wait_warp(smem_u32(&bar_main_full[chunk & 1]), (chunk >> 1) & 1, abortp, 64)) {
          ok = false;
          break;
        }
        tc_fence_after();
        promote_main_double(acc, taddr + (chunk & 1) * kDoubleCols, c == 0);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_main_free[chunk & 1]));
      }
      if (!ok) break;
      if constexpr (kEc) {
        if (!mbar_wait_warp(smem_u32(&bar_corr_full[tcount & 1]), (tcount >> 1) & 1, abortp, 64)) {
          ok = false;
          break;
        }
        tc_fence_after();
        fold_correction_double(acc, taddr + 256 + (tcount & 1) * kDoubleCols, kTf32 ? 1.0f : (1.0f / 2048.0f));
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_corr_free[tcount & 1]));
      }
      if constexpr (kSplit) {
        // to the CTA that stores this block; four columns of the 32 rows are 512 consecutive bytes
        const int per = Cfg::EPI_WARPS / parts;
        const uint32_t to = map_to_cta(smem_base + Cfg::PARTS_OFFSET + (part * per + ew % per) * Cfg::PART_BYTES + lane * 16, ew / per);
#pragma unroll
        for (int i = 0; i < Cfg::NC; i += 4) st_cluster_v4(to + i * 128, acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
      } else {
        store_narrow_block<Cfg>(acc, p, tc, BN, q, col_in, smem_gen, ew, lane);
      }
    }
    if (!ok) {
      abort_flag = 1;
      if (lane == 0) atomicCAS(p.status, 0, kErrEpilogueWait);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, Cfg::TMEM_COLS);
  if constexpr (kSplit) {
    // A CTA whose wait ran out has no part: it tells the others, and none of them stores its share of the tile.
    if (static_cast<int>(threadIdx.x) < parts && *abortp) raise_abort_in(&abort_flag, threadIdx.x);
    __syncwarp();
    cluster_sync_all();  // every part, or word that one is missing, has arrived
    const int ew = warp - 4, per = Cfg::EPI_WARPS / parts;
    if (warp >= 4 && ew / per == part && !*abortp) {
      const TileCoord tc = decode_tile(first_tile, p.tiles_m, p.tiles_n, Cfg::GROUP_M);
      const float4* from = reinterpret_cast<const float4*>(smem_gen + Cfg::PARTS_OFFSET + ew % per * Cfg::PART_BYTES) + lane;
      float acc[Cfg::NC];
#pragma unroll
      for (int i = 0; i < Cfg::NC; i += 4) {
        const float4 v = from[i * 8];
        acc[i] = v.x;
        acc[i + 1] = v.y;
        acc[i + 2] = v.z;
        acc[i + 3] = v.w;
      }
      for (int r = 1; r < parts; ++r) {
        from += per * (Cfg::PART_BYTES / 16);
#pragma unroll
        for (int i = 0; i < Cfg::NC; i += 4) {
          const float4 v = from[i * 8];
          acc[i] += v.x;
          acc[i + 1] += v.y;
          acc[i + 2] += v.z;
          acc[i + 3] += v.w;
        }
      }
      store_narrow_block<Cfg>(acc, p, tc, BN, warp & 3, (ew >> 2) * Cfg::NC, smem_gen, ew, lane);
    }
  }
}

}  // namespace tcec_sm100
