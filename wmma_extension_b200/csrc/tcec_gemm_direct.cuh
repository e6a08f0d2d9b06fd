// One-launch error-corrected GEMM on tcgen05 for batches of small and middle-sized matrices and for tiny calls:
// loader warps read the FP32 operands from global memory with ordinary loads, split them in registers and write
// the hi and lo operand images to a ring in shared memory; two threads issue the products; epilogue warps promote,
// fold and store.  No split pass, no workspace and no tensor maps, so any layout, leading dimension, alignment,
// batch stride and pointer table qualifies.
//
// Same split, same products in the same order, same promotion interval as the panel kernels
// (tcec_gemm_panels.cuh), so the same bits.
//
// What bounds it: HBM for small matrices (a 64^3 product moves 48 KB and does 1.6 MFLOP on the tensor pipe), the
// path from L2 and shared-memory bandwidth for larger ones (per K block 32 KB of images written and 48 KB read by
// the MMAs = 640 of the 128-byte cycles, against 384 tensor cycles).  What the split pass cost instead: operands read, written as
// panels padded to 256 rows, and read again; a 64^3 matrix took four times its own bytes in each direction.
//
// Several small matrices share a tile.  With S = 64 or 32 >= max(m, n), 128 / S matrices lie on the diagonal of one
// 128 x 128 tile: matrix p takes rows and columns p*S..; the off-diagonal products are computed and not
// read.  (An M = 128, N = 128 MMA takes 64 cycles and an N = 64 one 48, so the waste is cheaper than
// tiles of their own.)  Rows and columns beyond a matrix hold whatever the ring held: every element of D depends on
// its own row of A and column of B only, and those elements are not stored.  K is padded with zeros.
//
// Image of one operand and stage: 16-byte chunk c of row r at c * kLbo + r * 16 (un-swizzled K-major core matrices,
// 8-row groups 128 bytes apart).  kLbo is 2048 + 32, not 2048: with rows whose K is contiguous a store instruction
// covers the four chunks of a few rows, which the 32 bytes spread over all banks.
//
// Roles (640 threads, one persistent CTA per SM; registers re-balanced with setmaxnreg):
//   warp 1       one thread: main products; the main accumulator is double-buffered, so the products of a promotion
//                chunk run while the epilogue drains the one before
//   warp 2       one thread: correction products; double-buffered by tile
//   warps 4-11   epilogue (lane quarter = warp % 4, column half = (warp - 4) / 4)
//   warps 12-19  loaders: each holds two granules (K = 32, 16 registers per operand) in flight, across
//                tile boundaries, i.e. up to 64 KB per SM
#pragma once
#include "sm100_ptx.cuh"
#include "tcec_epilogue.cuh"
#include "tcec_gemm_panels.cuh"
#include "tcec_gemm_roles.cuh"
#include "tcec_panels.cuh"

namespace tcec_sm100 {

struct DirectOperand {
  const float* base;          // strided batch base (used when array == nullptr)
  const float* const* array;  // optional: one pointer per matrix
  long long ld, batch_stride;
  int rows;                   // extent along M (A) or N (B)
  int k_contiguous;           // element (r, k) at r*ld + k, else at k*ld + r
};

struct GemmDirectParams {
  DirectOperand a, b;
  int M, N, K, batch;
  int slot, slot_log2;    // S: 128, 64 or 32 rows (and columns) per matrix of a tile
  int tiles_m, tiles_n;   // 128 x 128 tiles per matrix (1 x 1 when slot < 128)
  int ntiles;
  int promo;              // K blocks per round-to-nearest promotion; 0 = once, at the end
  float alpha, beta;
  float* c;
  float* const* c_array;
  long long ldc, c_batch_stride;
  int c_col_major;
  int* status;
  int debug_flags;  // develop builds only: bit 6 = the first stage after the first ring fill is never filled
};

template <bool kTf32, bool kEc>
struct GemmDirectCfg {
  static constexpr int KOP = kTf32 ? 16 : 32;           // K per stage (one K block)
  static constexpr int kLbo = 128 * 16 + 32;
  static constexpr int IMAGE = 4 * kLbo;                 // one operand, hi or lo
  static constexpr int NP = kEc ? 2 : 1;
  static constexpr int STAGE = 2 * NP * IMAGE;           // A hi (lo), B hi (lo)
  static constexpr int NST = kEc ? 5 : 8;
  static constexpr int EPI_WARPS = 8, LOAD_WARPS = 8;
  static constexpr int EPI_OFFSET = NST * STAGE;
  static constexpr int SMEM_BYTES = NST * STAGE + EPI_WARPS * kEpiBufBytes + 128;
  static constexpr int THREADS = 128 + 32 * (EPI_WARPS + LOAD_WARPS);
  static constexpr int REGS_LAUNCH = 96, REGS_CONTROL = 32, REGS_EPILOGUE = 112, REGS_LOAD = 112;
  static_assert(128 * REGS_CONTROL + 32 * EPI_WARPS * REGS_EPILOGUE + 32 * LOAD_WARPS * REGS_LOAD <= THREADS * REGS_LAUNCH,
                "register shares exceed the launch allocation");
  static_assert(THREADS * REGS_LAUNCH <= 65536, "launch allocation exceeds the register file");
  static constexpr int TMEM_COLS = kEc ? 512 : 256;      // main x 2, corr x 2
};


__device__ __forceinline__ void st_shared_u4(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void st_shared_u2(uint32_t addr, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void st_shared_u1(uint32_t addr, uint32_t x) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(x) : "memory");
}

// One loader warp's view of one operand of the current tile.
//   rows contiguous: 16 units of 32 rows x 8 k; this warp takes units 2w and 2w+1 (row group u % 4, k chunk u / 4),
//                    lane = row, so every load is 128 contiguous bytes
//   K contiguous:    this warp takes rows 16w .. 16w+15; 16-byte loads (8 lanes = 128 bytes of a row, four rows per
//                    load) where the pointer and ld allow it, else pairs of k (16 lanes = 32 k of a row)
// Lanes whose row (or matrix) does not exist read one that does, so that a full granule needs no predicates on rows.
struct LoaderOperand {
  const float* p;   // first element this lane reads in granule 0 (rows contiguous: of unit 2w)
  const float* p1;  // rows contiguous: of unit 2w+1
  int rows;         // K contiguous: rows left from the lane's first row on (at least 1)
  bool vec4;        // K contiguous: 16-byte loads
};

template <bool kKc>
__device__ __forceinline__ void loader_setup(LoaderOperand& v, const DirectOperand& o, int first_matrix, int batch,
                                             int slot_log2, int row_tile, int w, int lane) {
  const int in_slot = (1 << slot_log2) - 1;
  if constexpr (!kKc) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int u = 2 * w + i, r = (u & 3) * 32 + lane, chunk = u >> 2;
      const int matrix = min(first_matrix + (r >> slot_log2), batch - 1), row = min(row_tile + (r & in_slot), o.rows - 1);
      const float* base = o.array ? o.array[matrix] : o.base + matrix * o.batch_stride;
      base = after_wait(base) + static_cast<long long>(chunk * 8) * o.ld + row;
      if (i == 0) v.p = base;
      else v.p1 = base;
    }
  } else {
    const int r0 = w * 16, matrix = min(first_matrix + (r0 >> slot_log2), batch - 1), row0 = row_tile + (r0 & in_slot);
    const float* base = after_wait(o.array ? o.array[matrix] : o.base + matrix * o.batch_stride);
    v.vec4 = o.ld % 4 == 0 && (reinterpret_cast<uintptr_t>(base) & 15) == 0;
    const int r = min(row0 + (v.vec4 ? lane >> 3 : lane >> 4), o.rows - 1);
    v.rows = o.rows - r;
    v.p = base + static_cast<long long>(r) * o.ld + (v.vec4 ? (lane & 7) * 4 : (lane & 15) * 2);
  }
}

// Reads this warp's 512 elements of one operand, k0 .. k0+31 (zeros beyond K).  kFull: all 32 exist.
template <bool kKc, bool kFull>
__device__ __forceinline__ void loader_read(float (&v)[16], const LoaderOperand& o, long long ld, int k0, int K, int w,
                                            int lane) {
  if constexpr (!kKc) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int kleft = K - k0 - ((2 * w + i) >> 2) * 8;
      const float* q = (i == 0 ? o.p : o.p1) + static_cast<long long>(k0) * ld;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        v[8 * i + e] = (kFull || e < kleft) ? ld_operand(q) : 0.f;
        q += ld;
      }
    }
  } else if (o.vec4) {
    const int kleft = K - k0 - (lane & 7) * 4;
    const float* q = o.p + k0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i == 0 || 4 * i < o.rows) {
        if (kFull || kleft >= 4) {
          t = ld_operand(reinterpret_cast<const float4*>(q));
        } else {
          if (kleft > 0) t.x = ld_operand(q);
          if (kleft > 1) t.y = ld_operand(q + 1);
          if (kleft > 2) t.z = ld_operand(q + 2);
        }
      }
      v[4 * i] = t.x;
      v[4 * i + 1] = t.y;
      v[4 * i + 2] = t.z;
      v[4 * i + 3] = t.w;
      q += 4 * ld;
    }
  } else {
    const int kleft = K - k0 - (lane & 15) * 2;
    const float* q = o.p + k0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const bool row = i == 0 || 2 * i < o.rows;
      v[2 * i] = (row && (kFull || kleft > 0)) ? ld_operand(q) : 0.f;
      v[2 * i + 1] = (row && (kFull || kleft > 1)) ? ld_operand(q + 1) : 0.f;
      q += 2 * ld;
    }
  }
}

// Splits what loader_read returned and writes it into the operand's images: chunks 0..3 of a row at `img0`, chunks
// 4..7 (tf32: the granule's second K block, where `two` says there is one) at `img1`; the lo image follows the hi image
// by Cfg::IMAGE.
template <bool kTf32, bool kEc, bool kKc>
__device__ __forceinline__ void loader_write(const float (&v)[16], bool vec4, uint32_t img0, uint32_t img1, bool two, int w,
                                             int lane) {
  using Cfg = GemmDirectCfg<kTf32, kEc>;
  if constexpr (!kKc) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int u = 2 * w + i;
      const uint32_t row = ((u & 3) * 32 + lane) * 16;
      if constexpr (kTf32) {
        if ((u >> 2) >= 2 && !two) continue;
        const uint32_t at = ((u >> 2) < 2 ? img0 : img1) + static_cast<uint32_t>(((u >> 2) & 1) * 2 * Cfg::kLbo) + row;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float x[4] = {v[8 * i + 4 * h], v[8 * i + 4 * h + 1], v[8 * i + 4 * h + 2], v[8 * i + 4 * h + 3]};
          uint4 hi, lo;
          split4_tf32(x, hi, lo);
          st_shared_u4(at + h * Cfg::kLbo, hi);
          if constexpr (kEc) st_shared_u4(at + h * Cfg::kLbo + Cfg::IMAGE, lo);
        }
      } else {
        uint4 hi, lo;
        split2_f16(v[8 * i], v[8 * i + 1], hi.x, lo.x);
        split2_f16(v[8 * i + 2], v[8 * i + 3], hi.y, lo.y);
        split2_f16(v[8 * i + 4], v[8 * i + 5], hi.z, lo.z);
        split2_f16(v[8 * i + 6], v[8 * i + 7], hi.w, lo.w);
        const uint32_t at = img0 + static_cast<uint32_t>((u >> 2) * Cfg::kLbo) + row;
        st_shared_u4(at, hi);
        if constexpr (kEc) st_shared_u4(at + Cfg::IMAGE, lo);
      }
    }
  } else if (vec4) {
    const int q = lane & 7;  // float4 of the row's granule
    const uint32_t row = (w * 16 + (lane >> 3)) * 16;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (kTf32) {
        if (q >= 4 && !two) continue;
        const float x[4] = {v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]};
        uint4 hi, lo;
        split4_tf32(x, hi, lo);
        const uint32_t at = (q < 4 ? img0 : img1) + (q & 3) * Cfg::kLbo + row + i * 64;
        st_shared_u4(at, hi);
        if constexpr (kEc) st_shared_u4(at + Cfg::IMAGE, lo);
      } else {
        uint32_t h0, h1, l0, l1;
        split2_f16(v[4 * i], v[4 * i + 1], h0, l0);
        split2_f16(v[4 * i + 2], v[4 * i + 3], h1, l1);
        const uint32_t at = img0 + (q >> 1) * Cfg::kLbo + (q & 1) * 8 + row + i * 64;
        st_shared_u2(at, h0, h1);
        if constexpr (kEc) st_shared_u2(at + Cfg::IMAGE, l0, l1);
      }
    }
  } else {
    const int j = lane & 15;  // pair of k
    const uint32_t row = (w * 16 + (lane >> 4)) * 16;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if constexpr (kTf32) {
        if (j >= 8 && !two) continue;
        const float h0 = tf32_rna(v[2 * i]), h1 = tf32_rna(v[2 * i + 1]);
        const uint32_t at = (j < 8 ? img0 : img1) + ((j & 7) >> 1) * Cfg::kLbo + (j & 1) * 8 + row + i * 32;
        st_shared_u2(at, __float_as_uint(h0), __float_as_uint(h1));
        if constexpr (kEc)
          st_shared_u2(at + Cfg::IMAGE, __float_as_uint(tf32_rna(v[2 * i] - h0)), __float_as_uint(tf32_rna(v[2 * i + 1] - h1)));
      } else {
        uint32_t hi, lo;
        split2_f16(v[2 * i], v[2 * i + 1], hi, lo);
        const uint32_t at = img0 + (j >> 2) * Cfg::kLbo + (j & 3) * 4 + row + i * 32;
        st_shared_u1(at, hi);
        if constexpr (kEc) st_shared_u1(at + Cfg::IMAGE, lo);
      }
    }
  }
}

struct DirectTile {
  int matrix, mt, nt;  // first matrix; tile position inside it (slot == 128)
};
__device__ __forceinline__ DirectTile direct_tile(const GemmDirectParams& p, int tile) {
  DirectTile t;
  if (p.slot < 128) {
    t.matrix = tile << (7 - p.slot_log2);
    t.mt = t.nt = 0;
  } else {
    const int per = p.tiles_m * p.tiles_n;
    t.matrix = tile / per;
    const int r = tile - t.matrix * per;
    t.mt = r / p.tiles_n;
    t.nt = r - t.mt * p.tiles_n;
  }
  return t;
}

// kAk, kBk: K is contiguous in A, in B (one loader path per kernel: with all of them in one, warps waited for
// instructions more than for anything else).  NC = columns per epilogue warp: 64 (slot 128) or 32 (slots 64 and 32).
template <bool kTf32, bool kEc, bool kAk, bool kBk, int NC>
__global__ void __launch_bounds__(GemmDirectCfg<kTf32, kEc>::THREADS, 1) tcec_gemm_direct_kernel(const GemmDirectParams p) {
  using Cfg = GemmDirectCfg<kTf32, kEc>;
  constexpr int NST = Cfg::NST;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[NST], bar_empty[NST];
  __shared__ uint64_t bar_main_full[2], bar_main_free[2], bar_corr_full[2], bar_corr_free[2], bar_drain[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ uint32_t abort_flag;

  const uint32_t smem_base = (smem_u32(smem_raw) + 127u) & ~127u;
  uint8_t* const smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int nkb = (p.K + Cfg::KOP - 1) / Cfg::KOP;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(smem_u32(&bar_full[s]), Cfg::LOAD_WARPS);
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
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;  // main buffers at +0 and +128, correction buffers at +256 and +384
  volatile uint32_t* abortp = &abort_flag;
  let_next_launch_start();
  wait_for_launch_before();

  if (warp >= 12) {
    // ------------------------------------------------------------ loaders
    setmaxnreg_inc<Cfg::REGS_LOAD>();
    const int w = warp - 12;
    const int ngran = (p.K + 31) / 32;
    // what is read next: granule `rg` of tile `rtile`
    int rtile = blockIdx.x, rg = 0;
    LoaderOperand oa, ob;
    auto setup = [&]() {
      const DirectTile t = direct_tile(p, rtile);
      loader_setup<kAk>(oa, p.a, t.matrix, p.batch, p.slot_log2, t.mt * 128, w, lane);
      loader_setup<kBk>(ob, p.b, t.matrix, p.batch, p.slot_log2, t.nt * 128, w, lane);
    };
    // From a tile to the CTA's next one a lane's pointers move by one and the same step in a strided batch of matrices of one tile,
    // as long as the tile is full and 16-byte loads stay aligned: six instructions instead of a hundred per tile, in a kernel whose
    // warps wait for instructions.  16384 x 64^3 172 -> 165 us, 10000 x 50 x 40 x 100 190 -> 179, 4096 x 128^3 176 -> 171.  (A third
    // granule in flight, i.e. half as much loader code again, cost 16384 x 64^3 170 -> 198.)
    const int members = 128 >> p.slot_log2, full_tiles = p.batch >> (7 - p.slot_log2);
    const bool steady = p.tiles_m * p.tiles_n == 1 && !p.a.array && !p.b.array &&
                        (!kAk || p.a.ld % 4 != 0 || p.a.batch_stride % 4 == 0) && (!kBk || p.b.ld % 4 != 0 || p.b.batch_stride % 4 == 0);
    const long long step_a = static_cast<long long>(gridDim.x) * members * p.a.batch_stride;
    const long long step_b = static_cast<long long>(gridDim.x) * members * p.b.batch_stride;
    auto next_tile = [&]() {
      rtile += gridDim.x;
      if (rtile >= p.ntiles) return;
      if (steady && rtile < full_tiles) {
        oa.p += step_a;
        ob.p += step_b;
        if constexpr (!kAk) oa.p1 += step_a;
        if constexpr (!kBk) ob.p1 += step_b;
      } else {
        setup();
      }
    };
    auto read = [&](float (&va)[16], float (&vb)[16], int& vec4) {
      if (rtile >= p.ntiles) return;
      if (rg * 32 + 32 <= p.K) {
        loader_read<kAk, true>(va, oa, p.a.ld, rg * 32, p.K, w, lane);
        loader_read<kBk, true>(vb, ob, p.b.ld, rg * 32, p.K, w, lane);
      } else {
        loader_read<kAk, false>(va, oa, p.a.ld, rg * 32, p.K, w, lane);
        loader_read<kBk, false>(vb, ob, p.b.ld, rg * 32, p.K, w, lane);
      }
      vec4 = (kAk && oa.vec4 ? 1 : 0) | (kBk && ob.vec4 ? 2 : 0);
      if (++rg == ngran) {
        rg = 0;
        next_tile();
      }
    };
    uint32_t s = 0, ph = 0;
    [[maybe_unused]] uint32_t filled = 0;  // stages before the current one
    bool ok = true;
    auto next_stage = [&]() {
      ++filled;
      if (++s == static_cast<uint32_t>(NST)) {
        s = 0;
        ph ^= 1;
      }
    };
    auto stage_free = [&]() {
      if (!mbar_wait_warp(smem_u32(&bar_empty[s]), ph ^ 1, abortp, 0)) return false;
      mbar_try_wait(smem_u32(&bar_empty[s]), ph ^ 1);  // each lane observes the completed phase itself
      return true;
    };
    // writes granule `g` of the tile being written
    auto write = [&](const float (&va)[16], const float (&vb)[16], int vec4, int g) {
      if (!stage_free()) return false;
      const uint32_t s0 = s, img0 = smem_base + s * Cfg::STAGE;
      // injected stall (failure-path test)
      const bool leave0 = dev_flag(p.debug_flags, 64) && filled == static_cast<uint32_t>(NST);
      const bool leave1 = dev_flag(p.debug_flags, 64) && filled + 1 == static_cast<uint32_t>(NST);
      uint32_t img1 = img0, s1 = s;
      bool two = false;
      next_stage();
      if constexpr (kTf32) {
        // a granule is two K blocks; the last one of a tile may have only one
        two = g * 2 + 1 < nkb;
        if (two) {
          if (!stage_free()) return false;
          s1 = s;
          img1 = smem_base + s * Cfg::STAGE;
          next_stage();
        }
      }
      loader_write<kTf32, kEc, kAk>(va, vec4 & 1, img0, img1, two, w, lane);
      loader_write<kTf32, kEc, kBk>(vb, vec4 >> 1, img0 + Cfg::NP * Cfg::IMAGE, img1 + Cfg::NP * Cfg::IMAGE, two, w, lane);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (!leave0) mbar_arrive(smem_u32(&bar_full[s0]));
        if (two && !leave1) mbar_arrive(smem_u32(&bar_full[s1]));
      }
      return true;
    };
    float a0[16], b0[16], a1[16], b1[16];
    int vec0 = 0, vec1 = 0;
    if (rtile < p.ntiles) setup();
    read(a0, b0, vec0);
    read(a1, b1, vec1);
    int wg = 0;  // granule being written
    for (int tile = blockIdx.x; tile < p.ntiles && ok;) {
      if (!write(a0, b0, vec0, wg)) {
        ok = false;
        break;
      }
      read(a0, b0, vec0);
      if (++wg == ngran) {
        wg = 0;
        tile += gridDim.x;
        if (tile >= p.ntiles) break;
      }
      if (!write(a1, b1, vec1, wg)) {
        ok = false;
        break;
      }
      read(a1, b1, vec1);
      if (++wg == ngran) {
        wg = 0;
        tile += gridDim.x;
      }
    }
    if (!ok) {
      abort_flag = 1;
      if (lane == 0) atomicCAS(p.status, 0, kErrProducerWait);
    }
  } else if (warp < 4) {
    setmaxnreg_dec<Cfg::REGS_CONTROL>();
    // ------------------------------------------------------------ MMA issuers
    if ((warp == 1 || (kEc && warp == 2)) && elect_one()) {
      DoubleImage im;
      im.dconst = umma_desc_kmajor_noswizzle(0, Cfg::kLbo, 128);
      im.base16 = (smem_base & 0x3ffff) >> 4;
      im.stage16 = Cfg::STAGE >> 4;
      im.a_lo16 = Cfg::IMAGE >> 4;
      im.b_hi16 = (Cfg::NP * Cfg::IMAGE) >> 4;
      im.b_lo16 = im.b_hi16 + (Cfg::IMAGE >> 4);
      im.kstep16 = (2 * Cfg::kLbo) >> 4;
      im.a_block16 = im.b_block16 = 0;
      int tile = static_cast<int>(blockIdx.x) - static_cast<int>(gridDim.x);
      auto next_tile = [&](uint32_t& idesc) {
        tile += gridDim.x;
        if (tile >= p.ntiles) return false;
        const int cols = p.slot < 128 ? 128 : min(128, (p.N - direct_tile(p, tile).nt * 128 + 15) & ~15);
        idesc = umma_idesc(kTf32 ? 2u : 0u, 128, cols);
        return true;
      };
      const KWalk walk{nkb, p.promo};
      const RingBarriers ring{bar_full, bar_empty};
      const bool ok = warp == 1 ? issue_main_double<kTf32, NST, 1>(next_tile, walk, im, tmem, ring, bar_main_full, bar_main_free, abortp)
                                : issue_corr_double<kTf32, NST, 1>(next_tile, walk, im, tmem + 256, ring, bar_corr_full,
                                                                   bar_corr_free, abortp);
      if (!ok) mma_thread_gave_up<false>(&abort_flag, p.status, kErrMmaWait, &bar_drain[warp - 1]);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    setmaxnreg_inc<Cfg::REGS_EPILOGUE>();
    const int ew = warp - 4, q = warp & 3, half = ew >> 2;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    // tile rows 32q.. belong to matrix `member` of the tile, whose columns start at member * slot
    const int member = (q * 32) >> p.slot_log2;
    const int row_in = q * 32 - member * p.slot;                       // of the matrix (tile) for lane 0
    const int col_in = p.slot == 32 ? 0 : half * NC;                   // likewise, for the warp's first column
    const bool idle = p.slot == 32 && half == 1;                       // 32 columns: one warp's worth
    const uint32_t taddr = tmem + lane_addr + member * p.slot + col_in;
    const int nchunks = p.promo ? (nkb + p.promo - 1) / p.promo : 1;
    uint32_t chunk = 0, tcount = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < p.ntiles && ok; tile += gridDim.x, ++tcount) {
      const DirectTile t = direct_tile(p, tile);
      float acc[NC];
      for (int c = 0; c < nchunks; ++c, ++chunk) {
        if (!mbar_wait_warp(smem_u32(&bar_main_full[chunk & 1]), (chunk >> 1) & 1, abortp, 0)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (!idle) promote_main_double(acc, taddr + (chunk & 1) * 128, c == 0);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_main_free[chunk & 1]));
      }
      if (!ok) break;
      if constexpr (kEc) {
        if (!mbar_wait_warp(smem_u32(&bar_corr_full[tcount & 1]), (tcount >> 1) & 1, abortp, 0)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (!idle) fold_correction_double(acc, taddr + 256 + (tcount & 1) * 128, kTf32 ? 1.0f : (1.0f / 2048.0f));
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_corr_free[tcount & 1]));
      }
      const int matrix = t.matrix + member;
      if (idle || matrix >= p.batch) continue;
      StoreTarget st;
      st.cbase = p.c_array ? p.c_array[matrix] : p.c + matrix * p.c_batch_stride;
      st.ldc = p.ldc;
      st.M = p.M;
      st.N = p.N;
      st.col_major = p.c_col_major;
      st.vec_ok = !p.c_col_major && (p.ldc % 4 == 0) && ((reinterpret_cast<uintptr_t>(st.cbase) & 15) == 0);
      st.alpha = p.alpha;
      st.beta = p.beta;
      const int row0 = t.mt * 128 + row_in, col0 = t.nt * 128 + col_in;
      if (row0 < p.M && col0 < p.N)
        store_warp_block<false, true>(acc, row0, col0, st, reinterpret_cast<float*>(smem_gen + Cfg::EPI_OFFSET) + ew * kEpiBufFloats, lane);
    }
    if (!ok) {
      abort_flag = 1;
      if (lane == 0) atomicCAS(p.status, 0, kErrEpilogueWait);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, Cfg::TMEM_COLS);
}

}  // namespace tcec_sm100
