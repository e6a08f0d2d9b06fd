// The panel GEMM on CTA pairs (tcgen05 cta_group::2): two SMs share one 256 x 256 output tile.
//
// Same arithmetic, panel format, roles and TMEM layout as tcec_gemm_panels.cuh.  What changes:
// each CTA of a pair loads the A panels of its own 128 rows and only its half of the B panels
// (128 of the tile's 256 N rows), and the leader CTA issues every MMA for both SMs
// (M = 256, N = 256, K = 16): per SM and K block 32 KB instead of 48 KB come through L2 and
// 48 KB instead of 72 KB of operands are read from shared memory, and the ring holds 6 stages
// instead of 4.  What bounds it at large sizes is the board's power (1000 W): the SM clock settles where the MMAs, the operands'
// way through L2 and the panels' way from DRAM add up to it.  16384^3 without copies takes 16.4 ms; with them 22.3 as long as the
// pairs drift apart along K (51.7 GB read from DRAM) and 19.3 with the pairs kept together (Pace, below: 19.2 GB, 16 if every wave
// read each of its panels once).
//
// Pair protocol (rank 0 = leader, rank 1 = peer):
//   full[s]   leader's barrier: its own copies' bytes + one remote arrive by the peer's relay
//             thread (peer warp 1), which waits on the peer's local full[s] first.  The remote
//             arrive has CTA scope: with cluster-scope release every arrive waited for the
//             SM's copies in flight and the ring degenerated to one stage at a time.
//   empty[s]  committed by the leader's two MMA threads to BOTH CTAs (multicast commit)
//   main_full / corr_full   likewise committed to both CTAs; each CTA drains its own TMEM
//   main_free / corr_free   leader's barriers: 8 local epilogue warps + 8 remote arrives
// Both CTAs meet at a cluster barrier after set-up and before exit.
//
// BN = 128 is the same kernel on 256 x 128 half tiles: a half is one 128-row B panel of which each
// CTA loads its 64 rows (the first or second 4 KB of the panel), multiplied with N = 128, and each
// epilogue warp holds 64 columns.  The host uses it for calls with so few tiles that whole tiles
// would leave at least half of the SM pairs idle (an N = 128 MMA takes ~0.6 of an N = 256 one, so
// halving pays only there); every element of C still sees the same products in the same order.
// A launch covers the pair tiles [tile_first, tile_first + tile_count).
#pragma once
#include "sm100_ptx.cuh"
#include "tcec_dispatch.h"
#include "tcec_gemm_panels.cuh"
#include "tcec_gemm_roles.cuh"

namespace tcec_sm100 {

template <bool kTf32, bool kEc>
struct GemmPairCfg {
  static constexpr int NP = kEc ? 2 : 1;
  static constexpr int KBS = stage_blocks(kEc);      // K blocks per stage
  static constexpr int BLOCK = kPanelBytes * NP;     // one K block of 128 rows: hi (+ lo)
  static constexpr int A_BYTES = BLOCK * KBS;        // this CTA's 128 rows of A
  static constexpr int B_BYTES = BLOCK * KBS;        // this CTA's 128 of the tile's 256 N rows
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int NST_RAW = (200 * 1024) / STAGE_BYTES;
  static constexpr int NST = NST_RAW > 8 ? 8 : NST_RAW;
  static constexpr int EPI_OFFSET = NST * STAGE_BYTES;
  static constexpr int SMEM_BYTES = NST * STAGE_BYTES + 8 * kEpiBufBytes + 1024;
  static constexpr int TMEM_COLS = kEc ? 512 : 256;
  static constexpr int THREADS = 384;
  // as in the one-SM kernel: the control warpgroup hands registers to the two epilogue warpgroups
  static constexpr int REGS_CONTROL = 40, REGS_EPILOGUE = 232;
  static_assert(128 * REGS_CONTROL + 256 * REGS_EPILOGUE <= THREADS * 168, "register shares");
  static constexpr int GROUP_M = tcec_host::kPairGroupM;  // pair tiles are 256 rows tall
};

// How the pairs of a launch share its tiles.  Strided: pair, pair + npairs, ...; with code for pacing (below) or without.  Drawn
// (and perhaps paced): from a device-wide counter, so that a pair that got its SMs late (another stream's kernel was there) takes
// fewer tiles instead of starting its whole share when the others are done: 8192 x 8192 x 4096 beside a kernel that holds four SMs
// 1890 us strided, 1200 drawn; alone 1210 and 1180.
enum PairTileMode : int { kStrided, kStridedPaced, kDrawn };

// Drawn tiles.  The leader's producer claims the next tile late in the one before, early enough for the counter's answer, and
// writes it, the end mark too, into a ring in either CTA, from which the other roles read.  An entry is one word, the tile and a bit
// that changes from round to round, so that nothing else has to be ordered with it; it is written again when all who read it, in
// either CTA, have arrived on its barrier in the leader.  Claimed only when it is needed, it
// kept the tensor pipe waiting for the counter (8192 x 8192 x 4096 2 % slower); claimed a whole tile ahead by a thread of its own, the pairs that
// start first took two tiles of the first wave, whose panels are then shared less (6000^3 10 % slower).
constexpr uint32_t kNoTile = 0x7fffffff;  // the end mark; tiles are below 2^31 - 1
struct DrawnTiles {
  const uint32_t* ring;   // this CTA's
  const uint64_t* empty;  // the barriers, of which the leader's are used
  uint32_t count = 0;
  // The index-th tile of this pair.  Whole warps read the entry in every lane: handed from one lane to the others it made every
  // promotion of the epilogue slower (10000 x 9500 x 1350 810 us, 717 so, 726 strided), by what ptxas then does with its registers.
  template <bool kWarp>
  __device__ __forceinline__ int at(uint32_t index, volatile uint32_t* abortp) const {
    const uint32_t slot = index % kTileRing, round = ~(index / kTileRing) & 1u;
    for (uint32_t i = 0; i < TCEC_WAIT_LIMIT; ++i) {
      const uint32_t v = ld_relaxed_cluster_own(smem_u32(ring + slot));
      const bool there = v >> 31 == round;
      if (kWarp ? __all_sync(0xffffffffu, there) : there) {
        if (!kWarp || (threadIdx.x & 31) == 0) mbar_arrive_cluster(map_to_cta(smem_u32(empty + slot), 0));
        return (v & kNoTile) == kNoTile ? static_cast<int>(kNoMoreTiles) : static_cast<int>(v & kNoTile);
      }
      __nanosleep(64);
      if ((i & 0xff) == 0xff && (kWarp ? __any_sync(0xffffffffu, *abortp != 0) : *abortp != 0)) break;
    }
    return kTileWaitFailed;
  }
  __device__ __forceinline__ int next(volatile uint32_t* abortp) { return at<false>(count++, abortp); }
  // The leader's producer: what it drew, to everybody.
  __device__ __forceinline__ int publish(unsigned int drawn, int ntiles, volatile uint32_t* abortp) {
    const bool more = drawn < static_cast<unsigned int>(ntiles);
    const uint32_t slot = count % kTileRing, round = ~(count / kTileRing) & 1u;
    if (!mbar_wait(smem_u32(empty + slot), round, abortp, 64)) return kTileWaitFailed;
    const uint32_t word = (more ? drawn : kNoTile) | round << 31;
    st_relaxed_cluster(map_to_cta(smem_u32(ring + slot), 1), word);
    st_relaxed_cluster(map_to_cta(smem_u32(ring + slot), 0), word);
    ++count;
    return more ? static_cast<int>(drawn) : static_cast<int>(kNoMoreTiles);
  }
};

// Keeps the pairs of a launch close together along K.  The pairs of a wave share their panels, each row block of A with the other
// tiles of its row and each of B with those of its column, and a panel comes from DRAM once if all of them read it while it is in
// L2.  Left alone they drift apart, tile after tile, until most panels are fetched several times.
// Every kPaceStages stages the leader's producer raises its count.  A thread of its own (the producer has no time for a round
// trip to L2: 16384^3 without correction 8.0 ms that way, 7.3 this way) adds it to a device-wide sum and holds the producer while
// its count is more than one above the mean of the pairs that have started: one whose SMs another kernel has taken must not stop the
// rest, and one that starts when the others are well under way counts from where they are.  A hold is bounded, and whoever has held
// in vain holds no more.
// 16384^3: 21.4 ms unpaced, 19.3 every 4 or 8 stages, 19.6 every 16; the words are a hint, results do not depend on them.
constexpr uint32_t kPaceStages = 8;
constexpr uint32_t kPaceLeft = 1u << 25;  // what a pair adds when it runs out of tiles, so that nobody waits for it
struct Pace {
  volatile uint32_t count, hold;  // shared memory; the producer writes `count` (kPaceLeft at its end), the pacing thread `hold`
};
__device__ __forceinline__ void pace_producer(Pace& pace, uint32_t count) {
  pace.count = count;
  for (int i = 0; i < 512 && pace.hold; ++i) __nanosleep(64);
}
// words[0]: the sum of the counts; words[1]: the pairs in it, each from its start on: from its first count on, those that start some
// microseconds before others did not wait for them (16384^3 without correction with the GPU hot 7.6 ms, 7.9 that way).
__device__ __forceinline__ void pace_launch(Pace& pace, unsigned int* words, uint32_t pairs, volatile uint32_t* abortp) {
  const uint32_t others = ld_relaxed_gpu(words + 1), mean = others ? ld_relaxed_gpu(words) / others : 0;
  if (mean >= kPaceLeft / 128) return;        // some have left
  const uint32_t base = mean > 16 ? mean : 0;  // pairs that the launch has SMs for start closer together
  atomicAdd(words + 1, 1u);
  if (base) atomicAdd(words, base);
  uint32_t added = 0;
  bool may_hold = true;
  for (uint32_t idle = 0; idle < TCEC_WAIT_LIMIT && !*abortp;) {
    const uint32_t count = pace.count;
    if (count == added) {
      __nanosleep(200);
      ++idle;
      continue;
    }
    idle = 0;
    uint32_t seen = atomicAdd(words, count - added) + (count - added);
    added = count;
    if (count >= kPaceLeft) return;
    const unsigned long long wanted_of_one = base + count - 1;
    if (!may_hold || seen >= wanted_of_one * pairs) continue;
    pace.hold = 1;
    const unsigned long long wanted = wanted_of_one * ld_relaxed_gpu(words + 1);  // all pairs, or fewer
    for (int i = 0; i < 128 && seen < wanted; ++i) {
      __nanosleep(200);
      seen = ld_relaxed_gpu(words);
    }
    may_hold = seen >= wanted;
    pace.hold = 0;
  }
  atomicAdd(words, kPaceLeft);
}

// p.tiles_m counts 256-row pair tiles here.  Without correction launches that are not paced have a kernel without it: the mere test in
// the producer's loop costs them 2 % (5000 x 6000 x 7000 460 us, 447).  With correction strided launches have one kernel, paced or
// not: apart, 4096^3 took 388.4 us instead of 385.7, complex 2048^3 207.2 instead of 204.7.  Drawing has a kernel of its own: as a
// choice at run time it cost the strided launches 4 % (4096^3 390, 407).
template <bool kTf32, bool kEc, int BN, int kMode>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(384, 1)
    tcec_gemm_panels_pair_kernel(const GemmPanelParams p) {
  constexpr bool kTilesDrawn = kMode == kDrawn;
  static_assert(BN == 256 || BN == 128, "whole or half-width pair tiles");
  using Cfg = GemmPairCfg<kTf32, kEc>;
  constexpr int NST = Cfg::NST;
  if (p.only_if) {
    wait_for_launch_before();
    if (*p.only_if == 0) return;
  }
  constexpr int HALVES = 256 / BN;            // work items per pair tile
  constexpr int NC = BN / 2;                  // columns per epilogue warp
  constexpr int B_PIECE = kPanelBytes / HALVES;  // bytes of one B image (hi or lo) per CTA and K block
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[NST], bar_empty[NST];
  __shared__ uint64_t bar_main_full, bar_main_free, bar_corr_full, bar_corr_free, bar_drain[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ uint32_t abort_flag;
  __shared__ Pace pace;
  __shared__ uint64_t bar_tile_empty[kTileRing];  // used in the leader only
  __shared__ uint32_t tile_ring[kTileRing];

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* const smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = (rank == 0);
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int ntiles = p.tile_count * HALVES;  // work items of this launch

  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(smem_u32(&bar_full[s]), leader ? 2 : 1);  // leader: own producer + the peer's relay
      mbar_init(smem_u32(&bar_empty[s]), kEc ? 2 : 1);
    }
    mbar_init(smem_u32(&bar_main_full), 1);
    mbar_init(smem_u32(&bar_main_free), 16);  // used in the leader only: 8 warps of each CTA
    mbar_init(smem_u32(&bar_corr_full), 1);
    mbar_init(smem_u32(&bar_corr_free), 16);
    mbar_init(smem_u32(&bar_drain[0]), 1);
    mbar_init(smem_u32(&bar_drain[1]), 1);
    abort_flag = 0;
    pace.count = pace.hold = 0;
    if constexpr (kTilesDrawn)
      for (int i = 0; i < kTileRing; ++i) {
        mbar_init(smem_u32(&bar_tile_empty[i]), (kEc ? 2 : 1) + 8 + 10);  // MMA threads and epilogue; the peer's producer, relay, epilogue
        tile_ring[i] = 0;
      }
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(&tmem_base_s), Cfg::TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_main = tmem_base_s;
  const uint32_t tmem_corr = tmem_base_s + 256;
  volatile uint32_t* abortp = &abort_flag;
  wait_for_launch_before();
  // What the leader's two MMA threads need (tcec_gemm_roles.cuh): M = 256 across the pair.
  OperandImage im;
  im.dconst = umma_desc_kmajor_noswizzle(0, 128, 512);
  im.base16 = (smem_base & 0x3ffff) >> 4;
  im.stage16 = Cfg::STAGE_BYTES >> 4;
  im.a_lo16 = kPanelBytes >> 4;
  im.b_hi16 = Cfg::A_BYTES >> 4;
  im.b_lo16 = (Cfg::A_BYTES + kPanelBytes) >> 4;
  im.idesc = umma_idesc(kTf32 ? 2u : 0u, 256, BN);
  im.a_block16 = im.b_block16 = Cfg::BLOCK >> 4;
  auto tiles = [&] {
    if constexpr (kTilesDrawn) return DrawnTiles{tile_ring, bar_tile_empty};
    else return StridedTiles{pair, npairs, ntiles};
  }();
  auto more = [&](int tile) { return kTilesDrawn ? tile >= 0 : tile < ntiles; };  // a failed wait for a drawn tile is no tile either
  const KWalk walk{p.nkb, p.promo};
  const RingBarriers ring{bar_full, bar_empty};

  if (warp < 4) {
    setmaxnreg_dec<Cfg::REGS_CONTROL>();
    if (warp == 0) {
      // ---------------------------------------------------------- producer (each CTA, own panels)
      if (elect_one()) {
        uint32_t s = 0, ph = 0, armed = 0, armed_parity = 0, it = 0;
        const bool paced = kMode != kStrided && p.pace && leader;  // the peer's ring cannot run ahead of the leader's
        bool ok = true;
        [[maybe_unused]] unsigned int drawn = kTilesDrawn && leader ? atomicAdd(&p.sched[0], 1u) : 0;
        [[maybe_unused]] const int claim_kb = p.nkb > 2 * NST * Cfg::KBS ? (p.nkb / Cfg::KBS - 2 * NST) * Cfg::KBS : 0;
        auto drawn_tile = [&] {
          if constexpr (kTilesDrawn) return leader ? tiles.publish(drawn, ntiles, abortp) : tiles.next(abortp);
          else return 0;
        };
        int tile = kTilesDrawn ? drawn_tile() : pair;
        for (; more(tile) && ok; tile = kTilesDrawn ? drawn_tile() : tile + npairs) {
          const TileCoord tc = decode_tile(p.tile_first + tile / HALVES, p.tiles_m, p.tiles_n, Cfg::GROUP_M);
          const uint8_t* pa = p.panels_a + tc.b * p.panels_a_batch_stride +
                              static_cast<size_t>(tc.mt * 2 + rank) * p.nkb * Cfg::BLOCK;
          // whole tile: this CTA's 128-row panel of the tile's two; half: its 64 rows of the half's one panel
          const int nblock = tc.nt * 2 + (BN == 256 ? static_cast<int>(rank) : tile % HALVES);
          const uint8_t* pb = p.panels_b + tc.b * p.panels_b_batch_stride +
                              static_cast<size_t>(nblock) * p.nkb * Cfg::BLOCK + (BN == 256 ? 0u : rank * B_PIECE);
          const int arows = panel_rows(p.M, tc.mt * 256 + static_cast<int>(rank) * 128);
          const int brows = BN == 256 ? panel_rows(p.N, nblock * 128) : 128;
          for (int kb = 0; kb < p.nkb; kb += Cfg::KBS, ++it) {
            if (!mbar_wait(smem_u32(&bar_empty[s]), ph ^ 1, abortp, 128)) {
              ok = false;
              break;
            }
            if (paced && it % kPaceStages == 0) pace_producer(pace, it / kPaceStages);
            if (kTilesDrawn && kb == claim_kb && leader) drawn = atomicAdd(&p.sched[0], 1u);
            if (dev_flag(p.debug_flags, 1) && it >= static_cast<uint32_t>(NST)) {  // develop builds: no loads
              mbar_arrive(smem_u32(&bar_full[s]));
              if (++s == static_cast<uint32_t>(NST)) {
                s = 0;
                ph ^= 1;
              }
              continue;
            }
            // injected stall (failure-path test): the first stage after the first ring fill is never filled
            if (dev_flag(p.debug_flags, 32) && it == static_cast<uint32_t>(NST)) {
              if (++s == static_cast<uint32_t>(NST)) {
                s = 0;
                ph ^= 1;
              }
              continue;
            }
            const uint32_t full = smem_u32(&bar_full[s]);
            const uint32_t dst = smem_base + s * Cfg::STAGE_BYTES;
            const int nblk = Cfg::KBS == 1 ? 1 : min(Cfg::KBS, p.nkb - kb);  // K blocks in this stage
            mbar_arrive_expect_tx(full, static_cast<uint32_t>(nblk) * Cfg::NP * (arows * 64 + (BN == 256 ? brows * 64 : B_PIECE)));
            armed |= 1u << s;
            armed_parity = (armed_parity & ~(1u << s)) | (ph << s);
            const uint8_t* srca = pa + static_cast<size_t>(kb) * Cfg::BLOCK;
            if (arows == 128) bulk_load(dst, srca, nblk * Cfg::BLOCK, full);
            else load_panel_rows(dst, srca, nblk * Cfg::NP, arows, full);
            const uint8_t* srcb = pb + static_cast<size_t>(kb) * Cfg::BLOCK;
            if constexpr (BN == 256) {
              if (brows == 128) bulk_load(dst + Cfg::A_BYTES, srcb, nblk * Cfg::BLOCK, full);
              else load_panel_rows(dst + Cfg::A_BYTES, srcb, nblk * Cfg::NP, brows, full);
            } else {
#pragma unroll
              for (int i = 0; i < Cfg::KBS; ++i)
                if (i < nblk)
#pragma unroll
                  for (int h = 0; h < Cfg::NP; ++h)  // hi (+ lo): each image keeps its place in the stage
                    bulk_load(dst + Cfg::A_BYTES + i * Cfg::BLOCK + h * kPanelBytes, srcb + i * Cfg::BLOCK + h * kPanelBytes,
                              B_PIECE, full);
            }
            if (++s == static_cast<uint32_t>(NST)) {
              s = 0;
              ph ^= 1;
            }
          }
        }
        if (paced) pace.count = kPaceLeft;
        if (kTilesDrawn && tile == kTileWaitFailed) ok = false;
        if (!ok) {
          raise_abort_pair(&abort_flag);
          atomicCAS(p.status, 0, kErrProducerWait);
          for (uint32_t q = 0; q < static_cast<uint32_t>(NST); ++q)
            if (armed & (1u << q)) mbar_wait_plain(smem_u32(&bar_full[q]), (armed_parity >> q) & 1);
        }
      }
    } else if (warp == 1) {
      if (elect_one()) {
        if (!leader) {
          // -------------------------------------------------------- peer: relay "my stage landed"
          uint32_t s = 0, ph = 0, it = 0;
          bool ok = true;
          int tile = kTilesDrawn ? tiles.next(abortp) : pair;
          for (; more(tile) && ok; tile = kTilesDrawn ? tiles.next(abortp) : tile + npairs) {
            for (int kb = 0; kb < p.nkb; kb += Cfg::KBS, ++it) {
              if (!mbar_wait(smem_u32(&bar_full[s]), ph, abortp, 32)) {
                ok = false;
                break;
              }
              mbar_arrive_cluster(map_to_cta(smem_u32(&bar_full[s]), 0));
              if (++s == static_cast<uint32_t>(NST)) {
                s = 0;
                ph ^= 1;
              }
            }
          }
          if (kTilesDrawn && tile == kTileWaitFailed) ok = false;
          if (!ok) {
            raise_abort_pair(&abort_flag);
            atomicCAS(p.status, 0, kErrMmaWait);
          }
        } else {
          // -------------------------------------------------------- leader: main products
          if (!issue_main_products<kTf32, true, NST, Cfg::KBS>(tiles, walk, im, tmem_main, ring, &bar_main_full,
                                                          &bar_main_free, abortp, p.debug_flags,
                                                                    blockIdx.x == 0 ? p.trace : nullptr))
            mma_thread_gave_up<true>(&abort_flag, p.status, kErrMmaWait, &bar_drain[0]);
        }
      }
    } else if (warp == 2) {
      // ---------------------------------------------------------- leader: correction products
      if constexpr (kEc) {
        if (leader && elect_one()) {
          if (!issue_corr_products<kTf32, true, NST>(tiles, walk, im, tmem_corr, ring, &bar_corr_full, &bar_corr_free,
                                                     abortp, p.debug_flags, blockIdx.x == 0 ? p.trace : nullptr))
            mma_thread_gave_up<true>(&abort_flag, p.status, kErrMmaWait, &bar_drain[1]);
        }
      }
    } else if (kMode != kStrided && p.pace && leader && elect_one()) {
      // ---------------------------------------------------------- leader: pacing
      pace_launch(pace, p.pace, static_cast<uint32_t>(npairs), abortp);
    }
  } else {
    // ------------------------------------------------------------ epilogue (each CTA, its 128 rows)
    setmaxnreg_inc<Cfg::REGS_EPILOGUE>();
    const int ew = warp - 4;
    const int q = warp & 3;
    const int colbase = (ew >> 2) * NC;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    const float corr_scale = kTf32 ? 1.0f : (1.0f / 2048.0f);
    const bool vec_store = !p.c_col_major && (p.ldc % 4 == 0);
    const uint32_t main_free_leader = map_to_cta(smem_u32(&bar_main_free), 0);
    const uint32_t corr_free_leader = map_to_cta(smem_u32(&bar_corr_free), 0);
    uint32_t chunk = 0, tcount = 0;
    bool ok = true;
    int tile = pair;
    for (; (kTilesDrawn || tile < ntiles) && ok; tile += kTilesDrawn ? 0 : npairs, ++tcount) {
      TileCoord tc{};
      if constexpr (kTilesDrawn) {
        tile = tiles.template at<true>(tcount, abortp);
        if (tile < 0) break;
      } else {
        tc = decode_tile(p.tile_first + tile / HALVES, p.tiles_m, p.tiles_n, Cfg::GROUP_M);
      }
      const int nchunks = p.promo ? (p.nkb + p.promo - 1) / p.promo : 1;
      float acc[NC];
      for (int c = 0; c < nchunks; ++c, ++chunk) {
        if (!mbar_wait_warp(smem_u32(&bar_main_full), chunk & 1, abortp)) {
          ok = false;
          break;
        }
        if (warp == 4 && lane == 0) trace_mark(p, 2, chunk);
        tc_fence_after();
        if constexpr (BN == 256) promote_main_chunk<true>(acc, tmem_main + lane_addr + colbase, c == 0);
        else promote_main_chunk(acc, tmem_main + lane_addr + colbase, c == 0);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(main_free_leader);
        if (warp == 4 && lane == 0) trace_mark(p, 3, chunk);
      }
      if (!ok) break;
      if constexpr (kEc) {
        if (!mbar_wait_warp(smem_u32(&bar_corr_full), tcount & 1, abortp)) {
          ok = false;
          break;
        }
        tc_fence_after();
      }
      if constexpr (kTilesDrawn) tc = decode_tile(p.tile_first + tile / HALVES, p.tiles_m, p.tiles_n, Cfg::GROUP_M);
      float* cbase = p.c_array ? p.c_array[tc.b] : p.c + tc.b * p.c_batch_stride;
      const int col0 = tc.nt * 256 + (tile % HALVES) * BN + colbase;
      const bool vec_ok = vec_store && ((reinterpret_cast<uintptr_t>(cbase) & 15) == 0);
      if constexpr (kEc) {
        fold_correction(acc, tmem_corr + lane_addr + colbase, corr_scale);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(corr_free_leader);
      }
      StoreTarget st;
      st.cbase = cbase;
      st.ldc = p.ldc;
      st.M = p.M;
      st.N = p.N;
      st.col_major = p.c_col_major;
      st.vec_ok = vec_ok;
      st.alpha = p.alpha;
      st.beta = p.beta;
      store_warp_block<true>(acc, tc.mt * 256 + static_cast<int>(rank) * 128 + q * 32, col0, st, reinterpret_cast<float*>(smem_gen + Cfg::EPI_OFFSET) + ew * kEpiBufFloats, lane);
    }
    if (kTilesDrawn && tile == kTileWaitFailed) ok = false;
    if (!ok) {
      raise_abort_pair(&abort_flag);
      if (lane == 0) atomicCAS(p.status, 0, kErrEpilogueWait);
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves while the other may still signal it or read its operands
  if (warp == 1) tmem_dealloc_pair(tmem_base_s, Cfg::TMEM_COLS);
  if (kTilesDrawn && leader && threadIdx.x == 0) {
    // Every pair has drawn its end mark by now; the last one out leaves the counters at zero.
    __threadfence();
    if (atomicAdd(&p.sched[1], 1u) == static_cast<unsigned int>(npairs) - 1) {
      p.sched[0] = 0;
      p.sched[1] = 0;
      __threadfence();
    }
  }
}

}  // namespace tcec_sm100
