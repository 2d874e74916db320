// Device building blocks shared by the block-sparse GEMM kernels:
//   * cp.async tile loader (16-byte chunks, zero fill for out-of-range parts)
//   * warp-level tile product: mma.sync m16n8k16 (FP16 / BF16, FP32 accumulate)
//     fed by ldmatrix, or FFMA for FP32 operands
//   * accumulator -> (row, col, value) iteration for the epilogues
//
// Shared-memory tiles keep the orientation the operand has in global memory,
// so that every copy is a plain 16-byte cp.async:
//   "K-contiguous"  tile[nonK][K]   pitch = TK + PAD
//   "K-strided"     tile[K][nonK]   pitch = extent + PAD
// PAD is 16 bytes, which makes the pitch an odd multiple of 16 bytes: eight
// consecutive rows fall into eight different 16-byte bank groups, so ldmatrix
// and the FP32 reads are conflict free.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace bsp {

template <typename T> struct Elem;
template <> struct Elem<float> { static constexpr int VEC = 4; static constexpr bool MMA = false; };
template <> struct Elem<__half> { static constexpr int VEC = 8; static constexpr bool MMA = true; };
template <> struct Elem<__nv_bfloat16> { static constexpr int VEC = 8; static constexpr bool MMA = true; };

template <typename T> __device__ __forceinline__ T cvt_out(float v);
template <> __device__ __forceinline__ float cvt_out<float>(float v) { return v; }
template <> __device__ __forceinline__ __half cvt_out<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 cvt_out<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// 2^x on the special-function unit (ex2.approx: about 2 ulp, denormals flushed).
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// 16-byte asynchronous copy; copies nothing and zero-fills when !pred.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool pred) {
  const int n = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(smem)), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Copies a tile of ROWS x CONT elements (CONT along the unit-stride direction
// of global memory) into shared memory with row pitch PITCH.  Rows >= rows_ok
// and columns >= cont_ok are zero-filled; `src` always stays a valid address.
template <typename T, int ROWS, int CONT, int PITCH, int NTHREADS>
__device__ __forceinline__ void load_tile(T* smem, const T* src, int64_t row_stride, int tid,
                                          int rows_ok, int cont_ok) {
  constexpr int VEC = Elem<T>::VEC;
  constexpr int CPR = CONT / VEC;            // chunks per row
  constexpr int TOTAL = ROWS * CPR;
#pragma unroll
  for (int it = 0; it < (TOTAL + NTHREADS - 1) / NTHREADS; ++it) {
    const int ch = tid + it * NTHREADS;
    if (TOTAL % NTHREADS == 0 || ch < TOTAL) {
      const int r = ch / CPR, c = (ch % CPR) * VEC;
      const bool ok = r < rows_ok && c < cont_ok;
      cp_async16(smem + r * PITCH + c, ok ? src + r * row_stride + c : src, ok);
    }
  }
}

// ---------------------------------------------------------------------------
// Warp tile product.  A is the [M][K] operand, B the [K][N] operand; AKC / BKC
// say whether their shared-memory tiles are K-contiguous.  The accumulator
// layout differs between the two back-ends; use for_each_acc to walk it.
// ---------------------------------------------------------------------------
template <typename T, int WM, int WN> struct Acc {
  static constexpr int COUNT = WM * WN / 32;
  float v[COUNT];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < COUNT; ++i) v[i] = 0.f;
  }
};

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

template <typename T>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma16816<__half>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma16816<__nv_bfloat16>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// FP32: which of the warp tile's rows (columns) accumulator index i of lane group g holds, of LANES groups
// with CNT rows each.  A K-contiguous operand is read 16 (8) bytes along K at a time, rows LANES apart
// (their pitch, an odd multiple of 16 bytes, spreads them over all banks); a K-strided one V = 4 or
// 2 consecutive rows at a time.  Single floats took one shared-memory instruction per operand value
// (batch 2, 4 heads, 1024^3, density 0.25, us: sdd block 16 / 32 / 64 / 128 with A transposed 303 -> 199,
// 160 -> 129, 144 -> 109, 123 -> 109; dsd transposed 179 -> 157, 148 -> 112, 132 -> 109, 150 -> 136).
// !WIDE: single floats, rows LANES apart, in either orientation (see kWide of sdd_impl.cuh).
template <bool KC, int LANES, int CNT, bool WIDE>
__device__ __forceinline__ constexpr int f32_index(int g, int i) {
  constexpr int V = CNT % 4 == 0 ? 4 : 2;
  return KC || !WIDE ? g + LANES * i : (i / V) * (LANES * V) + g * V + i % V;
}
// The CNT values of an operand at k0 .. k0 + KQ - 1: v[i][kk].
template <bool KC, int LANES, int CNT, int PITCH, int KQ, bool WIDE>
__device__ __forceinline__ void f32_load(const float* s, int base, int g, int k0, float (&v)[CNT][KQ]) {
  if constexpr (KC) {
#pragma unroll
    for (int i = 0; i < CNT; ++i) {
      const float* p = s + (base + g + LANES * i) * PITCH + k0;
      if constexpr (KQ == 4) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w;
      } else if constexpr (KQ == 2) {
        const float2 x = *reinterpret_cast<const float2*>(p);
        v[i][0] = x.x; v[i][1] = x.y;
      } else {
        v[i][0] = *p;
      }
    }
  } else if constexpr (!WIDE) {
#pragma unroll
    for (int kk = 0; kk < KQ; ++kk)
#pragma unroll
      for (int i = 0; i < CNT; ++i) v[i][kk] = s[(k0 + kk) * PITCH + base + g + LANES * i];
  } else {
    constexpr int V = CNT % 4 == 0 ? 4 : 2;
    static_assert(CNT % V == 0, "rows per lane");
#pragma unroll
    for (int kk = 0; kk < KQ; ++kk)
#pragma unroll
      for (int i = 0; i < CNT; i += V) {
        const float* p = s + (k0 + kk) * PITCH + base + f32_index<false, LANES, CNT, true>(g, i);
        if constexpr (V == 4) {
          const float4 x = *reinterpret_cast<const float4*>(p);
          v[i][kk] = x.x; v[i + 1][kk] = x.y; v[i + 2][kk] = x.z; v[i + 3][kk] = x.w;
        } else {
          const float2 x = *reinterpret_cast<const float2*>(p);
          v[i][kk] = x.x; v[i + 1][kk] = x.y;
        }
      }
  }
}

// One K-chunk (TK elements) of the warp tile at rows [m0, m0+WM), cols [n0, n0+WN).
// As / Bs point at the CTA tiles of the current stage; PA / PB are their pitches.
template <typename T, int WM, int WN, int TK, bool AKC, bool BKC, int PA, int PB, bool WIDE = true>
__device__ __forceinline__ void warp_tile_mma(Acc<T, WM, WN>& acc, const T* As, const T* Bs,
                                              int m0, int n0, int lane) {
  if constexpr (Elem<T>::MMA) {
    constexpr int MI = WM / 16, NI = WN / 8;
    static_assert(WM % 16 == 0 && WN % 16 == 0 && TK % 16 == 0, "mma tile shape");
    const int l7 = lane & 7, mi4 = lane >> 3;
#pragma unroll
    for (int k0 = 0; k0 < TK; k0 += 16) {
      uint32_t a[MI][4];
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const int mb = m0 + i * 16;
        if constexpr (AKC) {
          // matrices: (m+0,k+0) (m+8,k+0) (m+0,k+8) (m+8,k+8)
          ldsm_x4(a[i], smem_u32(As + (mb + (mi4 & 1) * 8 + l7) * PA + k0 + (mi4 >> 1) * 8));
        } else {
          // stored [k][m]: same four matrices, read transposed
          ldsm_x4_t(a[i], smem_u32(As + (k0 + (mi4 >> 1) * 8 + l7) * PA + mb + (mi4 & 1) * 8));
        }
      }
#pragma unroll
      for (int j = 0; j < NI; j += 2) {
        const int nb = n0 + j * 8;
        uint32_t b[4];
        if constexpr (BKC) {
          // stored [n][k]; matrices: (n+0,k+0) (n+0,k+8) (n+8,k+0) (n+8,k+8)
          ldsm_x4(b, smem_u32(Bs + (nb + (mi4 >> 1) * 8 + l7) * PB + k0 + (mi4 & 1) * 8));
        } else {
          // stored [k][n]; same four matrices, read transposed
          ldsm_x4_t(b, smem_u32(Bs + (k0 + (mi4 & 1) * 8 + l7) * PB + nb + (mi4 >> 1) * 8));
        }
#pragma unroll
        for (int i = 0; i < MI; ++i) {
          mma16816<T>(*reinterpret_cast<float(*)[4]>(&acc.v[(i * NI + j) * 4]), a[i], b[0], b[1]);
          mma16816<T>(*reinterpret_cast<float(*)[4]>(&acc.v[(i * NI + j + 1) * 4]), a[i], b[2], b[3]);
        }
      }
    }
  } else {
    // FP32: lane (ty, tx) = (lane / 4, lane % 4) owns RI rows and CJ columns (f32_index), k ascending.
    // (with 32 accumulators or more per thread, two values of k at a time leave registers for more warps;
    // 32 x 32 with only B K-contiguous: one, sdd block 32 takes 192 us with one, 222 with two, 214 with single floats)
    constexpr int RI = WM / 8, CJ = WN / 4, KQ = !WIDE || (!AKC && BKC && WM == 32 && WN == 32) ? 1 : RI * CJ >= 32 ? 2 : 4;
    static_assert(TK % 4 == 0 && PA % 4 == 0 && PB % 4 == 0, "16-byte reads");
    const int ty = lane >> 2, tx = lane & 3;
#pragma unroll
    for (int k = 0; k < TK; k += KQ) {
      float av[RI][KQ], bv[CJ][KQ];
      f32_load<AKC, 8, RI, PA, KQ, WIDE>(As, m0, ty, k, av);
      f32_load<BKC, 4, CJ, PB, KQ, WIDE>(Bs, n0, tx, k, bv);
#pragma unroll
      for (int kk = 0; kk < KQ; ++kk)
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
          for (int j = 0; j < CJ; ++j) acc.v[i * CJ + j] = fmaf(av[i][kk], bv[j][kk], acc.v[i * CJ + j]);
    }
  }
}

// Calls f(row, col, value) for every accumulator element of the warp tile
// (row / col relative to the warp tile origin).
template <typename T, int WM, int WN, bool AKC, bool BKC, bool WIDE = true, typename F>
__device__ __forceinline__ void for_each_acc(const Acc<T, WM, WN>& acc, int lane, F&& f) {
  if constexpr (Elem<T>::MMA) {
    constexpr int MI = WM / 16, NI = WN / 8;
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r)
          f(i * 16 + g + 8 * (r >> 1), j * 8 + 2 * t + (r & 1), acc.v[(i * NI + j) * 4 + r]);
  } else {
    constexpr int RI = WM / 8, CJ = WN / 4;
    const int ty = lane >> 2, tx = lane & 3;
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int j = 0; j < CJ; ++j) f(f32_index<AKC, 8, RI, WIDE>(ty, i), f32_index<BKC, 4, CJ, WIDE>(tx, j), acc.v[i * CJ + j]);
  }
}

}  // namespace bsp
