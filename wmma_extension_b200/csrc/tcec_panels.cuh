// Split pass of the panel path: FP32 matrix -> hi / scaled-lo operand panels.
//
// Follows the reference split (include/wmma_extension/tcec/tcec.hpp:219-223,
// scale include/wmma_extension/tcec/detail/scale.hpp:8-20):
//   hi = cast<T>(v);  lo = cast<T>((v - float(hi)) * s)
// with T = fp16 (round-to-nearest-even, s = 2^11) or tf32 (cvt.rna, s = 1).
// The reference redoes this in every warp that consumes a tile; here every
// element is split once and stored in the exact shared-memory image the
// tensor-core instruction reads, so the GEMM kernel moves panels with linear
// bulk copies and never touches the data with CUDA cores.
//
// Panel = 128 rows x 64 bytes of K (32 fp16 or 16 tf32), 8192 bytes, stored as
// un-swizzled K-major core matrices: element (r, c) with c a 16-byte chunk
// index 0..3 sits at (r/8)*512 + c*128 + (r%8)*16.  For each (row block, k
// block) the hi panel comes first and, with error correction, the lo panel
// directly after it.
#pragma once
#include <cuda_fp16.h>

#include <cstdint>

#include "sm100_ptx.cuh"

namespace tcec_sm100 {

constexpr int kPanelRows = 128;
constexpr int kPanelBytes = 8192;

__device__ __forceinline__ float tf32_rna(float v) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return __uint_as_float(r);
}

// 2 fp32 -> 2 packed fp16 hi and 2 packed fp16 scaled residuals.  The fp16 head is an operand of a mixed-precision
// multiply-add (h * -1 + v, exact) and both residuals are scaled in one packed multiplication: five instructions a
// pair instead of eight, and the same bits, signs of zeros included.
__device__ __forceinline__ void split2_f16(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 hv = __floats2half2_rn(x, y);
  hi = *reinterpret_cast<const uint32_t*>(&hv);
  float rx, ry;
  asm("{\n\t.reg .b16 l, u, m;\n\t.reg .b64 r, s;\n\t"
      "mov.b32 {l, u}, %2;\n\t"
      "mov.b16 m, 0xbc00;\n\t"
      "fma.rn.f32.f16 %0, l, m, %3;\n\t"
      "fma.rn.f32.f16 %1, u, m, %4;\n\t"
      "mov.b64 r, {%0, %1};\n\t"
      "mov.b64 s, {%5, %5};\n\t"
      "mul.rn.f32x2 r, r, s;\n\t"
      "mov.b64 {%0, %1}, r;\n\t}"
      : "=&f"(rx), "=&f"(ry)
      : "r"(hi), "f"(x), "f"(y), "f"(2048.0f));
  const __half2 lv = __floats2half2_rn(rx, ry);
  lo = *reinterpret_cast<const uint32_t*>(&lv);
}
// 8 fp32 -> 8 fp16 hi and 8 fp16 scaled residuals (16 bytes each).
__device__ __forceinline__ void split8_f16(const float (&v)[8], uint4& hi, uint4& lo) {
  split2_f16(v[0], v[1], hi.x, lo.x);
  split2_f16(v[2], v[3], hi.y, lo.y);
  split2_f16(v[4], v[5], hi.z, lo.z);
  split2_f16(v[6], v[7], hi.w, lo.w);
}
// 4 fp32 -> 4 tf32 hi and 4 tf32 residuals (16 bytes each).
__device__ __forceinline__ void split4_tf32(const float (&v)[4], uint4& hi, uint4& lo) {
  float h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    h[i] = tf32_rna(v[i]);
    l[i] = tf32_rna(v[i] - h[i]);
  }
  hi = make_uint4(__float_as_uint(h[0]), __float_as_uint(h[1]), __float_as_uint(h[2]),
                  __float_as_uint(h[3]));
  lo = make_uint4(__float_as_uint(l[0]), __float_as_uint(l[1]), __float_as_uint(l[2]),
                  __float_as_uint(l[3]));
}

struct SplitParams {
  const float* src;              // strided batch base (used when src_array == nullptr)
  const float* const* src_array; // optional pointer array, one matrix per batch entry
  long long ld;                  // leading dimension in elements
  long long batch_stride;        // elements between matrices (strided form)
  int rows;                      // extent along M (for A) or N (for B)
  int k;                         // extent along K
  int k_contiguous;              // 1: element (r,k) at r*ld + k ; 0: at k*ld + r
  int row_blocks;                // padded rows / 128
  int nkb;                       // number of k blocks
  uint8_t* panels;               // output
  long long panels_batch_stride; // bytes
  int skip_padding;              // 1: rows beyond the matrix are left as they are (they only reach elements of the product
                                 // that nobody stores); 0: they are written as zeros
};

// One CTA's work: the hi(+lo) panel of k block `kb`, row block `rb` of matrix `b`.
template <bool kTf32, bool kEc>
__device__ __forceinline__ void split_one_panel(const SplitParams& p, int kb, int rb, int b) {
  constexpr int KCH = kTf32 ? 4 : 8;    // fp32 elements per 16-byte operand chunk
  constexpr int KOP = 4 * KCH;          // K extent of one panel
  const float* src = after_wait(p.src_array ? p.src_array[b] : p.src + static_cast<long long>(b) * p.batch_stride);
  uint8_t* out = p.panels + static_cast<long long>(b) * p.panels_batch_stride +
                 (static_cast<size_t>(rb) * p.nkb + kb) * (kEc ? 2 : 1) * kPanelBytes;
  const int k0 = kb * KOP;
  const bool vec_ok = (p.ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(src) & 15) == 0);
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int item = threadIdx.x + it * 256;  // 512 (row, chunk) items per panel
    int r, c;
    if (p.k_contiguous) {
      r = item >> 2;
      c = item & 3;
    } else {
      r = item & 127;
      c = item >> 7;
    }
    const int row = rb * kPanelRows + r;
    if (p.skip_padding && row >= p.rows) continue;
    const int kk = k0 + c * KCH;
    float v[KCH];
    if (p.k_contiguous) {
      const float* s = src + static_cast<long long>(row) * p.ld + kk;
      if (row < p.rows && kk + KCH <= p.k && vec_ok) {
#pragma unroll
        for (int q = 0; q < KCH / 4; ++q) {
          const float4 t = ld_operand(reinterpret_cast<const float4*>(s) + q);
          v[4 * q + 0] = t.x;
          v[4 * q + 1] = t.y;
          v[4 * q + 2] = t.z;
          v[4 * q + 3] = t.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < KCH; ++q) v[q] = (row < p.rows && kk + q < p.k) ? ld_operand(s + q) : 0.f;
      }
    } else {
#pragma unroll
      for (int q = 0; q < KCH; ++q)
        v[q] = (row < p.rows && kk + q < p.k)
                   ? ld_operand(src + static_cast<long long>(kk + q) * p.ld + row)
                   : 0.f;
    }
    uint4 hi, lo;
    if constexpr (kTf32) {
      split4_tf32(v, hi, lo);
    } else {
      split8_f16(v, hi, lo);
    }
    const int off = (r >> 3) * 512 + c * 128 + (r & 7) * 16;
    *reinterpret_cast<uint4*>(out + off) = hi;
    if constexpr (kEc) *reinterpret_cast<uint4*>(out + kPanelBytes + off) = lo;
  }
}

// Split of one operand of a complex product into the panels of a real one of twice the K.  With K' = 2p + d and
// rows (plain, for A) or doubled rows (for B)
//   A'(i, 2p) = Re A(i, p),  A'(i, 2p + 1) = Im A(i, p)
//   B'(2j, 2p) = Re B(p, j), B'(2j, 2p + 1) = -Im B(p, j);  B'(2j + 1, 2p) = Im B(p, j), B'(2j + 1, 2p + 1) = Re B(p, j)
// column 2j of A' B' is the real part and column 2j + 1 the imaginary part of column j of A B: the real GEMM
// writes interleaved C.  Every complex element is read once; a doubled operand writes it into two rows.
struct ComplexSplitParams {
  const float* src;   // interleaved; 8-byte alignment is used where it is there, not required
  long long ld;       // complex elements
  int rows, k;        // complex extents
  int k_contiguous;   // element (r, p) at r*ld + p, else at p*ld + r
  int doubled;
  int nkb;            // K blocks of the panels
  uint8_t* panels;
};
template <bool kTf32, bool kEc>
__device__ __forceinline__ void split_complex_panel(const ComplexSplitParams& p, int kb, int rb) {
  constexpr int PC = kTf32 ? 2 : 4;  // complex elements per 16-byte operand chunk
  uint8_t* out = p.panels + (static_cast<size_t>(rb) * p.nkb + kb) * (kEc ? 2 : 1) * kPanelBytes;
  const int R = p.doubled ? 64 : 128;  // complex rows of this panel
  const float* const src = after_wait(p.src);
  const bool pairs = (reinterpret_cast<uintptr_t>(src) & 7) == 0;
  for (int item = threadIdx.x; item < R * 4; item += 256) {
    const int r = p.k_contiguous ? item >> 2 : item % R, c = p.k_contiguous ? item & 3 : item / R;
    const int row = rb * R + r, k0 = (kb * 4 + c) * PC;
    const long long step = p.k_contiguous ? 1 : p.ld;
    const float* q =
        src + 2 * (p.k_contiguous ? static_cast<long long>(row) * p.ld + k0 : static_cast<long long>(k0) * p.ld + row);
    float2 z[PC];
#pragma unroll
    for (int e = 0; e < PC; ++e) {
      const float* x = q + 2 * e * step;
      z[e] = make_float2(0.f, 0.f);
      if (row < p.rows && k0 + e < p.k) z[e] = pairs ? ld_operand(reinterpret_cast<const float2*>(x)) : make_float2(ld_operand(x), ld_operand(x + 1));
    }
    const int halves = p.doubled ? 2 : 1;
    for (int h = 0; h < halves; ++h) {
      const int orow = p.doubled ? 2 * r + h : r;
      float v[2 * PC];
#pragma unroll
      for (int e = 0; e < PC; ++e) {
        v[2 * e] = h ? z[e].y : z[e].x;
        v[2 * e + 1] = h ? z[e].x : (p.doubled ? -z[e].y : z[e].y);
      }
      uint4 hi, lo;
      if constexpr (kTf32) split4_tf32(v, hi, lo);
      else split8_f16(v, hi, lo);
      const int off = (orow >> 3) * 512 + c * 128 + (orow & 7) * 16;
      *reinterpret_cast<uint4*>(out + off) = hi;
      if constexpr (kEc) *reinterpret_cast<uint4*>(out + kPanelBytes + off) = lo;
    }
  }
}
// Both operands of a complex product: blocks below `panels_a` write A's panels.
template <bool kTf32, bool kEc>
__global__ void __launch_bounds__(256) tcec_split_complex_kernel(const ComplexSplitParams pa, const ComplexSplitParams pb,
                                                                 unsigned int panels_a) {
  let_next_launch_start();
  wait_for_launch_before();
  const bool second = blockIdx.x >= panels_a;
  const ComplexSplitParams& p = second ? pb : pa;
  const unsigned int i = second ? blockIdx.x - panels_a : blockIdx.x;
  split_complex_panel<kTf32, kEc>(p, i % p.nkb, i / p.nkb);
}

// grid = (nkb, row_blocks, batch), 256 threads: one CTA writes one hi(+lo) panel.
template <bool kTf32, bool kEc>
__global__ void __launch_bounds__(256) tcec_split_panels_kernel(const SplitParams p) {
  let_next_launch_start();
  wait_for_launch_before();
  split_one_panel<kTf32, kEc>(p, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Both operands of a product in one launch (grid.x = panels of A + panels of B, all matrices of the
// batch): one launch gap and one grid tail less than two launches, which is what a short call
// notices (4096^3: 3 of 361 us; 1024^3: 3 of 30).
template <bool kTf32, bool kEc>
__device__ __forceinline__ void split_panel_of_both(const SplitParams& pa, const SplitParams& pb, unsigned int panels_a,
                                                    unsigned int x) {
  const bool second = x >= panels_a;
  const SplitParams& p = second ? pb : pa;
  unsigned int i = second ? x - panels_a : x;
  const int kb = i % p.nkb;
  i /= p.nkb;
  const int rb = i % p.row_blocks;
  split_one_panel<kTf32, kEc>(p, kb, rb, static_cast<int>(i / p.row_blocks));
}
template <bool kTf32, bool kEc>
__global__ void __launch_bounds__(256) tcec_split_both_kernel(const SplitParams pa, const SplitParams pb,
                                                              unsigned int panels_a) {
  let_next_launch_start();
  wait_for_launch_before();
  split_panel_of_both<kTf32, kEc>(pa, pb, panels_a, blockIdx.x);
}

// The same behind a device word: gate[0] zero = the launch does nothing, for which its grid is small (eight CTAs per SM; a
// CTA per panel would take 20 us to do nothing at 32768 panels).  CTAs draw their panels two at a time from gate[1], zero
// before the launch: striding over them leaves SMs idle that were faster than others and spreads the accesses (4096 x
// 132^3 by tables with one matrix unaligned: 748 us strided, 668 drawn, 640 with a CTA per panel).
constexpr unsigned int kGatedPanels = 2;
template <bool kTf32, bool kEc>
__global__ void __launch_bounds__(256) tcec_split_both_gated_kernel(const SplitParams pa, const SplitParams pb,
                                                                    unsigned int panels_a, unsigned int panels,
                                                                    unsigned int* gate) {
  let_next_launch_start();
  wait_for_launch_before();
  if (*gate == 0) return;
  __shared__ unsigned int next[2];
  int turn = 0;
  for (unsigned int x = blockIdx.x * kGatedPanels; x < panels; turn ^= 1) {
    if (threadIdx.x == 0) next[turn] = (gridDim.x + atomicAdd(gate + 1, 1u)) * kGatedPanels;
    for (const unsigned int last = min(panels, x + kGatedPanels); x < last; ++x)
      split_panel_of_both<kTf32, kEc>(pa, pb, panels_a, x);
    __syncthreads();
    x = next[turn];
  }
}

}  // namespace tcec_sm100
