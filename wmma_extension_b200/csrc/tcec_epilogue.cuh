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

constexpr int kEpiBufFloats = 32 * 33;              // one warp's turn buffer
constexpr int kEpiBufBytes = kEpiBufFloats * 4;      // 4224

// `row0` = first of the warp's 32 rows (lane = row0 + lane holds `acc`), `col0` = first of its
// NC columns, `wbuf` = this warp's buffer of kEpiBufFloats floats.  Warp-collective.
//
// kWide: where every row of the block starts on a 32-byte boundary and C is not read, each lane stores its own row
// directly, a whole 32-byte sector per store, and leaves shared memory to the MMAs' operand reads.  Panel kernels
// (64 x 4096 x 4096 packed 34.8 -> 32.9 us, 2048^3 complex 216 -> 212, no other case slower); not the direct kernel, whose
// loads and stores share the path (16384 x 64^3 194 -> 204), nor the FP32-tile kernel, which stores through TMA.
template <bool kWide, int NC>
__device__ __forceinline__ void store_warp_block(const float (&acc)[NC], int row0, int col0, const StoreTarget& t,
                                                 float* wbuf, int lane) {
  // Old values of C a lane holds at once (beta != 0).  Read one before each store, every load waited for the store before it:
  // 1000 x 777 x 1111 with a column-major C and beta 26.6 us, in groups 20.5.  The kernels with fewer registers left
  // (kWide = false) stay with one: groups of 8 cost them 4096 x 128^3 195 -> 230 us without any beta.
  constexpr int kGroup = 16;
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
    } else {
#pragma unroll
      for (int g = 0; g < NC; g += kGroup) {
        const int left = t.N - col0 - g;
        float old[kGroup];
        float* q = dst;
#pragma unroll
        for (int i = 0; i < kGroup; ++i) {
          old[i] = (t.beta != 0.f && i < left) ? *q : 0.f;
          q += t.ldc;
        }
#pragma unroll
        for (int i = 0; i < kGroup; ++i) {
          if (i < left) *dst = t.beta != 0.f ? axpby(t.alpha, acc[g + i], t.beta, old[i]) : __fmul_rn(t.alpha, acc[g + i]);
          dst += t.ldc;
        }
      }
    }
    return;
  }
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
  const int rsub = lane >> 3, cv = (lane & 7) * 4;
#pragma unroll
  for (int cc = 0; cc < NC / 32; ++cc) {
#pragma unroll
    for (int i = 0; i < 32; ++i) wbuf[lane * 33 + i] = acc[cc * 32 + i];
    __syncwarp();
    if constexpr (kWide) {
      // in groups of row slices, so that a group's old values of C (beta != 0) are on their way together
#pragma unroll
      for (int part = 0; part < 8; part += kGroup / 4) {
        const int col = col0 + cc * 32 + cv;
        const bool vec = t.vec_ok && col + 3 < t.N;
        float4 old[kGroup / 4];
#pragma unroll
        for (int j = 0; j < kGroup / 4; ++j) {
          old[j] = make_float4(0.f, 0.f, 0.f, 0.f);
          const int row = row0 + (part + j) * 4 + rsub;
          if (t.beta != 0.f && row < t.M) {
            const float* src = t.cbase + static_cast<long long>(row) * t.ldc + col;
            if (vec) {
              old[j] = *reinterpret_cast<const float4*>(src);
            } else {
              if (col < t.N) old[j].x = src[0];
              if (col + 1 < t.N) old[j].y = src[1];
              if (col + 2 < t.N) old[j].z = src[2];
              if (col + 3 < t.N) old[j].w = src[3];
            }
          }
        }
#pragma unroll
        for (int j = 0; j < kGroup / 4; ++j) {
          const int r = (part + j) * 4 + rsub;
          const int row = row0 + r;
          const float* src = wbuf + r * 33 + cv;
          const float v0 = src[0], v1 = src[1], v2 = src[2], v3 = src[3];
          if (row < t.M) {
            float* dst = t.cbase + static_cast<long long>(row) * t.ldc + col;
            float4 o;
            if (t.beta != 0.f)
              o = make_float4(axpby(t.alpha, v0, t.beta, old[j].x), axpby(t.alpha, v1, t.beta, old[j].y),
                              axpby(t.alpha, v2, t.beta, old[j].z), axpby(t.alpha, v3, t.beta, old[j].w));
            else
              o = make_float4(__fmul_rn(t.alpha, v0), __fmul_rn(t.alpha, v1), __fmul_rn(t.alpha, v2), __fmul_rn(t.alpha, v3));
            if (vec) {
              *reinterpret_cast<float4*>(dst) = o;
            } else {
              if (col < t.N) dst[0] = o.x;
              if (col + 1 < t.N) dst[1] = o.y;
              if (col + 2 < t.N) dst[2] = o.z;
              if (col + 3 < t.N) dst[3] = o.w;
            }
          }
        }
      }
    } else {
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
    }
    __syncwarp();
  }
}

}  // namespace tcec_sm100
