// Second-order Taylor feature map for linear attention and its gradient, for sm_100a:
//     phi(x) = [1, x / d^(1/4), vec(x x^T) / (sqrt(2) sqrt(d))]        (1 + d + d^2 features)
// so that phi(q) . phi(k) = 1 + s + s^2 / 2 with s = q . k / sqrt(d). The reference has no such code
// (its README only links the idea); benchmark configuration 4 feeds these features, d = 16 -> 273,
// to LinearAttentionSmallVHD. The forward kernel writes the features straight into rows padded to
// a multiple of 8 elements, i.e. in the layout the attention kernels address with TMA, so no pad
// pass is needed; the backward kernel contracts the feature gradients back to d raw dimensions.
#pragma once
#include "fla_normalize.cuh"  // cp.async wrappers

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fla {

template <int D>
struct TaylorDims {
  static constexpr int F = 1 + D + D * D;        // features
  static constexpr int FP = (F + 7) / 8 * 8;     // padded row length (elements)
  static constexpr int PIECES = FP / 8;          // 16-byte pieces per row
};

__device__ __forceinline__ float taylor_c1(int d) { return rsqrtf(sqrtf(static_cast<float>(d))); }
__device__ __forceinline__ float taylor_c2(int d) { return rsqrtf(2.f * static_cast<float>(d)); }

constexpr int kTaylorRows = 128;  // rows per block tile (one thread per row) in both kernels
// Row stride of the staged feature tiles in 16-byte pieces: odd, so that one thread per row moving
// 16-byte pieces touches different banks in each quarter of a warp, and consecutive pieces of a row
// (the coalesced side) do too.
template <int D>
constexpr int kTaylorStride = TaylorDims<D>::PIECES | 1;
template <int D>
__host__ __device__ constexpr int taylor_tile_smem_bytes() {
  return kTaylorRows * kTaylorStride<D> * 16;
}

// x: [rows][D] bf16 contiguous; phi: [rows][FP] bf16 (FP - F zero columns at the end).
// Thread t computes the features of row t from registers (all indices are compile-time) into a
// shared-memory tile; the block then writes the tile out in coalesced 16-byte pieces.
template <int D>
__global__ void __launch_bounds__(kTaylorRows)
fla_taylor_fwd_kernel(const __nv_bfloat16* __restrict__ x, uint4* __restrict__ phi, long long rows) {
  using dims = TaylorDims<D>;
  static_assert(D % 8 == 0, "raw rows are moved as 16-byte pieces");
  extern __shared__ uint4 taylor_smem[];
  const float c1 = taylor_c1(D), c2 = taylor_c2(D);
  for (long long row0 = static_cast<long long>(blockIdx.x) * kTaylorRows; row0 < rows;
       row0 += static_cast<long long>(gridDim.x) * kTaylorRows) {
    const int nrows = static_cast<int>(min(static_cast<long long>(kTaylorRows), rows - row0));
    __syncthreads();  // the previous tile has been written out
    const int r = threadIdx.x;
    if (r < nrows) {
      float xv[D];
      const uint4* xrow = reinterpret_cast<const uint4*>(x + (row0 + r) * D);
#pragma unroll
      for (int pc = 0; pc < D / 8; ++pc) {
        const uint4 v = xrow[pc];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          xv[pc * 8 + 2 * j] = __uint_as_float(w[j] << 16);
          xv[pc * 8 + 2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
        }
      }
      uint4* out = taylor_smem + r * kTaylorStride<D>;
      auto feature = [&](int f) -> float {  // f is a compile-time constant after unrolling
        if (f == 0) return 1.f;
        if (f <= D) return c1 * xv[f - 1];
        if (f < dims::F) return c2 * xv[(f - 1 - D) / D] * xv[(f - 1 - D) % D];
        return 0.f;
      };
#pragma unroll
      for (int pc = 0; pc < dims::PIECES; ++pc) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const __nv_bfloat162 pr = __floats2bfloat162_rn(feature(8 * pc + 2 * j), feature(8 * pc + 2 * j + 1));
          w[j] = *reinterpret_cast<const uint32_t*>(&pr);
        }
        out[pc] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nrows * dims::PIECES; idx += kTaylorRows) {
      const int rr = idx / dims::PIECES, pc = idx - rr * dims::PIECES;
      phi[(row0 + rr) * dims::PIECES + pc] = taylor_smem[rr * kTaylorStride<D> + pc];
    }
  }
}

// dx[r][a] = c1 dphi[r][1 + a] + c2 sum_b (dphi[r][1 + D + a D + b] + dphi[r][1 + D + b D + a]) x[r][b]
// dphi: [rows][FP] bf16 (row stride FP), x: [rows][D] bf16, dx: [rows][D] bf16.
// A block stages kTaylorRows rows of dphi in shared memory with cp.async, every piece of the tile in
// flight at once, then thread t contracts row t, one 16-byte piece at a time. Bound by HBM (three
// blocks of 72 KB are resident per SM at D = 16, so one computes while the others load). 262,144
// rows: 53 us with scalar shared-memory stores of a synchronous load, 36 us now (147 MB).
template <int D>
__global__ void __launch_bounds__(kTaylorRows)
fla_taylor_bwd_kernel(const uint4* __restrict__ dphi, const __nv_bfloat16* __restrict__ x,
                      __nv_bfloat16* __restrict__ dx, long long rows) {
  using dims = TaylorDims<D>;
  extern __shared__ uint4 taylor_smem[];
  const float c1 = taylor_c1(D), c2 = taylor_c2(D);
  for (long long row0 = static_cast<long long>(blockIdx.x) * kTaylorRows; row0 < rows;
       row0 += static_cast<long long>(gridDim.x) * kTaylorRows) {
    const int nrows = static_cast<int>(min(static_cast<long long>(kTaylorRows), rows - row0));
    __syncthreads();  // the previous tile has been consumed
    for (int idx = threadIdx.x; idx < nrows * dims::PIECES; idx += kTaylorRows) {
      const int r = idx / dims::PIECES, pc = idx - r * dims::PIECES;
      cp_async16(norm_smem_u32(taylor_smem + r * kTaylorStride<D> + pc), dphi + (row0 + r) * dims::PIECES + pc);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int r = threadIdx.x;
    if (r < nrows) {
      static_assert(D % 8 == 0, "raw rows are moved as 16-byte pieces");
      float xv[D], acc[D];
      const uint4* xrow = reinterpret_cast<const uint4*>(x + (row0 + r) * D);
#pragma unroll
      for (int pc = 0; pc < D / 8; ++pc) {
        const uint4 v = xrow[pc];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          xv[pc * 8 + 2 * j] = __uint_as_float(w[j] << 16);
          xv[pc * 8 + 2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
        }
      }
#pragma unroll
      for (int a = 0; a < D; ++a) acc[a] = 0.f;
#pragma unroll
      for (int pc = 0; pc < dims::PIECES; ++pc) {
        const uint4 v = taylor_smem[r * kTaylorStride<D> + pc];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int f = 8 * pc + j;  // compile-time after unrolling, as are a and b
          const float gv = __uint_as_float((j & 1) ? (w[j >> 1] & 0xFFFF0000u) : (w[j >> 1] << 16));
          if (f >= 1 && f <= D) {
            acc[f - 1] += c1 * gv;
          } else if (f > D && f < dims::F) {
            const int a = (f - 1 - D) / D, b = (f - 1 - D) % D;
            acc[a] += c2 * gv * xv[b];
            acc[b] += c2 * gv * xv[a];
          }
        }
      }
      uint4* orow = reinterpret_cast<uint4*>(dx + (row0 + r) * D);
#pragma unroll
      for (int pc = 0; pc < D / 8; ++pc) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const __nv_bfloat162 pr = __floats2bfloat162_rn(acc[pc * 8 + 2 * j], acc[pc * 8 + 2 * j + 1]);
          w[j] = *reinterpret_cast<const uint32_t*>(&pr);
        }
        orow[pc] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
}

}  // namespace fla
