// Store step shared by the GEMM kernels: one epilogue thread holds NC (128, or 64 in half-width
// tiles) consecutive columns of one output row (main + correction already folded) and the warp writes alpha * acc + beta * C.
// Restates the reference's smem2dmem (test/tcec/batch_gemm.cu:119-185): beta == 0 never reads C,
// 128-bit stores where the row allows them, element-wise predicated stores on the ragged edge.
//
// A TMEM load leaves lane = row, so a direct store of a row-major C touches 32 different rows
// per instruction (32 partial sectors).  The warp therefore turns each 32 x 32 block through a
// private shared-memory buffer (pitch 33 floats: conflict-free both ways) and stores it as
// 4 rows x 128 contiguous bytes per instruction.  Column-major C needs no turn: consecutive
// lanes already hold consecutive addresses.
#pragma once
#include <cstdint>

#include "sm100_ptx.cuh"

namespace tcec_sm100 {

struct StoreTarget {
  float* cbase;      // first element of this matrix
  long long ldc;
  int M, N;
  int col_major;     // C(row, col) at col * ldc + row, else at row * ldc + col
  bool vec_ok;       // row-major, ldc % 4 == 0 and cbase 16-byte aligned
  float alpha, beta;
};

// alpha * v + beta * old with fixed rounding points (one product rounded, then one fused
// multiply-add), so every store path of every kernel produces the same bits.
__device__ __forceinline__ float axpby(float alpha, float v, float beta, float old) {
  return __fmaf_rn(beta, old, __fmul_rn(alpha, v));
}

__device__ __forceinline__ void st_global_v8(float* p, const float (&v)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]),
               "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

template <int NC>
__device__ __forceinline__ void store_row_slice(const float (&acc)[NC], int row, int col0, const StoreTarget& t) {
  if (row >= t.M) return;
#pragma unroll
  for (int cc = 0; cc < NC / 32; ++cc) {
    if (!t.col_major) {
      float* crow = t.cbase + static_cast<long long>(row) * t.ldc;
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const int col = col0 + cc * 32 + i;
        if (t.vec_ok && col + 3 < t.N) {
          float4 o;
          if (t.beta != 0.f) {
            const float4 old = *reinterpret_cast<const float4*>(crow + col);
            o.x = axpby(t.alpha, acc[cc * 32 + i + 0], t.beta, old.x);
            o.y = axpby(t.alpha, acc[cc * 32 + i + 1], t.beta, old.y);
            o.z = axpby(t.alpha, acc[cc * 32 + i + 2], t.beta, old.z);
            o.w = axpby(t.alpha, acc[cc * 32 + i + 3], t.beta, old.w);
          } else {
            o.x = __fmul_rn(t.alpha, acc[cc * 32 + i + 0]);
            o.y = __fmul_rn(t.alpha, acc[cc * 32 + i + 1]);
            o.z = __fmul_rn(t.alpha, acc[cc * 32 + i + 2]);
            o.w = __fmul_rn(t.alpha, acc[cc * 32 + i + 3]);
          }
          *reinterpret_cast<float4*>(crow + col) = o;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (col + e < t.N)
              crow[col + e] = t.beta != 0.f ? axpby(t.alpha, acc[cc * 32 + i + e], t.beta, crow[col + e])
                                            : __fmul_rn(t.alpha, acc[cc * 32 + i + e]);
          }
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int col = col0 + cc * 32 + i;
        if (col < t.N) {
          float* dst = t.cbase + static_cast<long long>(col) * t.ldc + row;
          *dst = t.beta != 0.f ? axpby(t.alpha, acc[cc * 32 + i], t.beta, *dst) : __fmul_rn(t.alpha, acc[cc * 32 + i]);
        }
      }
    }
  }
}

constexpr int kOldValues = 16;  // of C that a lane holds at once

template <int kVec>
__device__ __forceinline__ void store_updated(const float* src, float* dst, const float (&old)[kVec], const StoreTarget& t) {
  if constexpr (kVec == 4)
    *reinterpret_cast<float4*>(dst) = make_float4(axpby(t.alpha, src[0], t.beta, old[0]), axpby(t.alpha, src[1], t.beta, old[1]),
                                                  axpby(t.alpha, src[2], t.beta, old[2]), axpby(t.alpha, src[3], t.beta, old[3]));
  else
    *dst = axpby(t.alpha, src[0], t.beta, old[0]);
}
// A lane's part of a 32 x 32 block in the turn buffer: `all` pieces of kVec floats, the first `rows` of which are the matrix's,
// from `src` on every `src_step` floats to `dst` on every `dst_step`.  Old values of C are read kOldValues at a time, so that
// they are on their way together.
template <int kVec>
__device__ __forceinline__ void store_turned(const float* src, int src_step, float* dst, long long dst_step, int rows, int all,
                                             const StoreTarget& t) {
  constexpr int kGroup = kOldValues / kVec;
  if (rows > all) rows = all;
  if (t.beta == 0.f) {
#pragma unroll 4
    for (int r = 0; r < rows; ++r, src += src_step, dst += dst_step) {
      if constexpr (kVec == 4)
        *reinterpret_cast<float4*>(dst) = make_float4(__fmul_rn(t.alpha, src[0]), __fmul_rn(t.alpha, src[1]),
                                                      __fmul_rn(t.alpha, src[2]), __fmul_rn(t.alpha, src[3]));
      else
        *dst = __fmul_rn(t.alpha, src[0]);
    }
    return;
  }
#pragma unroll 1
  for (int left = rows; left > 0; left -= kGroup) {
    float old[kGroup][kVec];
    const float* q = dst;
#pragma unroll
    for (int g = 0; g < kGroup; ++g) {  // beyond the matrix: its last piece again, so that no load needs a predicate
      if constexpr (kVec == 4) {
        const float4 v = *reinterpret_cast<const float4*>(q);
        old[g][0] = v.x;
        old[g][1] = v.y;
        old[g][2] = v.z;
        old[g][3] = v.w;
      } else {
        old[g][0] = *q;
      }
      q += g + 1 < left ? dst_step : 0;
    }
#pragma unroll
    for (int g = 0; g < kGroup; ++g, src += src_step, dst += dst_step)
      if (g < left) store_updated<kVec>(src, dst, old[g], t);
  }
}

// The two ways below are the direct kernel's.  Its warps share the SM's instruction cache with loaders and MMA issuers and waited for
// instructions more than for anything else: they are short loops, with 32-bit shared addresses, and rows of C that are 16-byte
// aligned go through the buffer in 128-bit pieces.  us, unrolled with a predicate per element and like this: 16384 x 64^3 182, 171;
// 16384 x 32^3 72, 55; 4096 x 128^3 200, 183; 3000 x 127^3 217, 163; 2000 x 100^3 117, 94; one 32^3 6.4, 4.7.  The FP32-tile
// kernel, whose C leaves by TMA or column-major, gains nothing; the panel kernels, whose code would hold both ways four times,
// lose (300 x 201^3 87.2, 89.8).
// A lane's column of a 32 x 32 block in the turn buffer, row pitch 33 floats: `rows` rows of the matrix (at most 32), from `src`, to
// `dst` on every `ldc`.
__device__ __forceinline__ void store_column(uint32_t src, float* dst, int rows, const StoreTarget& t) {
  if (rows > 32) rows = 32;
  if (t.beta == 0.f) {
#pragma unroll 4
    for (int r = 0; r < rows; ++r, src += 132, dst += t.ldc) *dst = __fmul_rn(t.alpha, ld_shared_f32(src));
  } else {
#pragma unroll 1
    for (int r = 0; r < rows; ++r, src += 132, dst += t.ldc) *dst = axpby(t.alpha, ld_shared_f32(src), t.beta, *dst);
  }
}

// A whole 32-column block, `v` this lane's row of it, to `dst` (row 0, column 0 of the block), of which the matrix has `rows` rows.
// Eight 128-bit accesses of the buffer each way instead of 32 of 32 bits.
__device__ __forceinline__ void store_whole_block(const float* v, float* dst, int rows, const StoreTarget& t, uint32_t wbuf, int lane) {
  const uint32_t row = wbuf + lane * 128, turn = (lane & 7) << 4;
#pragma unroll
  for (int j = 0; j < 8; ++j) st_shared_v4(row + ((j << 4) ^ turn), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  __syncwarp();
  int r = lane >> 3;  // row r's piece p is at 128 r + 16 (p ^ r % 8); this lane's rows are r, r + 4, ...
  const int piece = lane & 7;
  dst += static_cast<long long>(r) * t.ldc + 4 * piece;
  const long long step = 4 * t.ldc;
  if (t.beta == 0.f) {
#pragma unroll 4
    for (int i = 0; i < 8; ++i, r += 4, dst += step) {
      const float4 x = ld_shared_v4(wbuf + r * 128 + ((piece ^ (r & 7)) << 4));
      if (r < rows)
        *reinterpret_cast<float4*>(dst) =
            make_float4(__fmul_rn(t.alpha, x.x), __fmul_rn(t.alpha, x.y), __fmul_rn(t.alpha, x.z), __fmul_rn(t.alpha, x.w));
    }
  } else {
#pragma unroll 1
    for (int i = 0; i < 8; ++i, r += 4, dst += step) {
      const float4 x = ld_shared_v4(wbuf + r * 128 + ((piece ^ (r & 7)) << 4));
      if (r < rows) {
        const float4 old = *reinterpret_cast<const float4*>(dst);
        *reinterpret_cast<float4*>(dst) = make_float4(axpby(t.alpha, x.x, t.beta, old.x), axpby(t.alpha, x.y, t.beta, old.y),
                                                      axpby(t.alpha, x.z, t.beta, old.z), axpby(t.alpha, x.w, t.beta, old.w));
      }
    }
  }
  __syncwarp();
}

constexpr int kEpiBufFloats = 32 * 33;              // one warp's turn buffer
constexpr int kEpiBufBytes = kEpiBufFloats * 4;      // 4224

// `row0` = first of the warp's 32 rows (lane = row0 + lane holds `acc`), `col0` = first of its
// NC columns, `wbuf` = this warp's buffer of kEpiBufFloats floats.  Warp-collective.
//
// kWide: where every row of the block starts on a 32-byte boundary and C is not read, each lane stores its own row
// directly, a whole 32-byte sector per store, and leaves shared memory to the MMAs' operand reads.  Panel kernels
// (64 x 4096 x 4096 packed 34.8 -> 32.9 us, 2048^3 complex 216 -> 212, no other case slower); not the direct kernel, whose
// loads and stores share the path (16384 x 64^3 194 -> 204), nor the FP32-tile kernel, which stores through TMA.
// kPieces: the direct kernel's stores of a row-major C (above).
template <bool kWide, bool kPieces = false, int NC>
__device__ __forceinline__ void store_warp_block(const float (&acc)[NC], int row0, int col0, const StoreTarget& t,
                                                 float* wbuf, int lane) {
  // Old values of C a lane holds at once (beta != 0).  Read one before each store, every load waited for the store before it:
  // 1000 x 777 x 1111 with a column-major C and beta 26.6 us, in groups 20.5.  The kernels with fewer registers left
  // (kWide = false) stay with one: groups of 8 cost them 4096 x 128^3 195 -> 230 us without any beta.
  constexpr int kGroup = kOldValues;
  if (kWide && t.vec_ok && t.beta == 0.f && col0 + NC <= t.N && t.ldc % 8 == 0 && (reinterpret_cast<uintptr_t>(t.cbase) & 31) == 0) {
    if (row0 + lane < t.M) {
      float* dst = t.cbase + static_cast<long long>(row0 + lane) * t.ldc + col0;
#pragma unroll
      for (int i = 0; i < NC; i += 8) {
        float o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = __fmul_rn(t.alpha, acc[i + e]);
        st_global_v8(dst + i, o);
      }
    }
    return;
  }
  if (t.col_major) {
    // Consecutive lanes hold consecutive addresses; one pointer walks the columns (multiplying and comparing per column
    // cost 256 x 512^3 by pointer tables 342 us instead of 289).
    if (row0 + lane >= t.M) return;
    float* dst = t.cbase + static_cast<long long>(col0) * t.ldc + row0 + lane;
    if (t.beta == 0.f && col0 + NC <= t.N) {
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        *dst = __fmul_rn(t.alpha, acc[i]);
        dst += t.ldc;
      }
      return;
    }
    if constexpr (!kWide) {
      store_row_slice(acc, row0 + lane, col0, t);
    } else if (t.beta == 0.f) {
      const int left = t.N - col0;
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        if (i < left) *dst = __fmul_rn(t.alpha, acc[i]);
        dst += t.ldc;
      }
    } else {
#pragma unroll
      for (int g = 0; g < NC; g += kGroup) {
        const int left = t.N - col0 - g;
        if (left > 0) {
          float old[kGroup];
          const float* q = dst;
#pragma unroll
          for (int i = 0; i < kGroup; ++i) {  // beyond the matrix: its last column again, so that no load needs a predicate
            old[i] = *q;
            q += i + 1 < left ? t.ldc : 0;
          }
#pragma unroll
          for (int i = 0; i < kGroup; ++i) {
            if (i < left) *dst = axpby(t.alpha, acc[g + i], t.beta, old[i]);
            dst += t.ldc;
          }
        }
      }
    }
    return;
  }
  if constexpr (kPieces) {
    const uint32_t turn = smem_u32(wbuf);
#pragma unroll
    for (int cc = 0; cc < NC / 32; ++cc) {
      const int first = col0 + cc * 32;
      if (first >= t.N) return;
      float* const dst = t.cbase + static_cast<long long>(row0) * t.ldc + first;
      if (t.vec_ok && first + 32 <= t.N) {
        store_whole_block(&acc[cc * 32], dst, t.M - row0, t, turn, lane);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) st_shared_f32(turn + lane * 132 + i * 4, acc[cc * 32 + i]);
        __syncwarp();
        if (first + lane < t.N) store_column(turn + lane * 4, dst + lane, t.M - row0, t);
        __syncwarp();
      }
    }
    return;
  }
  const int rsub = lane >> 3, cv = (lane & 7) * 4;
  if constexpr (kWide) {
    // Short loops, a uniform choice between them, and no predicate per element: with rows, edges and old values unrolled
    // and predicated together this part kept the warps waiting for instructions (592 x 128 x 200 x 16 on one-SM tiles 90 us,
    // like this 37; 12000 x 12001 x 1100 1150 and 890; 8192 x 8190 x 2048 830 and 720).
#pragma unroll
    for (int cc = 0; cc < NC / 32; ++cc) {
      const int first = col0 + cc * 32;
      if (first >= t.N) return;
#pragma unroll
      for (int i = 0; i < 32; ++i) wbuf[lane * 33 + i] = acc[cc * 32 + i];
      __syncwarp();
      if (t.vec_ok && first + 32 <= t.N) {
        // a row slice of four columns per lane, four rows apart
        store_turned<4>(wbuf + rsub * 33 + cv, 4 * 33, t.cbase + static_cast<long long>(row0 + rsub) * t.ldc + first + cv, 4 * t.ldc,
                        (t.M - row0 - rsub + 3) >> 2, 8, t);
      } else if (first + lane < t.N) {
        // a column per lane
        store_turned<1>(wbuf + lane, 33, t.cbase + static_cast<long long>(row0) * t.ldc + first + lane, t.ldc, t.M - row0, 32, t);
      }
      __syncwarp();
    }
  } else {
#pragma unroll
    for (int cc = 0; cc < NC / 32; ++cc) {
#pragma unroll
      for (int i = 0; i < 32; ++i) wbuf[lane * 33 + i] = acc[cc * 32 + i];
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int r = j * 4 + rsub;
        const int row = row0 + r, col = col0 + cc * 32 + cv;
        const float* src = wbuf + r * 33 + cv;
        const float v0 = src[0], v1 = src[1], v2 = src[2], v3 = src[3];
        if (row < t.M) {
          float* dst = t.cbase + static_cast<long long>(row) * t.ldc + col;
          if (t.vec_ok && col + 3 < t.N) {
            float4 o;
            if (t.beta != 0.f) {
              const float4 old = *reinterpret_cast<const float4*>(dst);
              o = make_float4(axpby(t.alpha, v0, t.beta, old.x), axpby(t.alpha, v1, t.beta, old.y),
                              axpby(t.alpha, v2, t.beta, old.z), axpby(t.alpha, v3, t.beta, old.w));
            } else {
              o = make_float4(__fmul_rn(t.alpha, v0), __fmul_rn(t.alpha, v1), __fmul_rn(t.alpha, v2),
                              __fmul_rn(t.alpha, v3));
            }
            *reinterpret_cast<float4*>(dst) = o;
          } else {
            const float v[4] = {v0, v1, v2, v3};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if (col + e < t.N)
                dst[e] = t.beta != 0.f ? axpby(t.alpha, v[e], t.beta, dst[e]) : __fmul_rn(t.alpha, v[e]);
            }
          }
        }
      }
      __syncwarp();
    }
  }
}

}  // namespace tcec_sm100
