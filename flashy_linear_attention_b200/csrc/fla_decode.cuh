// A few tokens from a running state, for sm_100a: the recurrence itself,
//     S += k_t^T v_t,   o_t = q_t S        (t = 0 .. tokens - 1)
// in fp32 on the CUDA cores (the reference has no counterpart: its kernels always start from an
// empty state and take multiples of 64 tokens, flashlinear/kernels/linear_attn_kernels.py:323-325).
//
// Bound by HBM: the state (dk x dv fp32, 64 KB a head at 128 x 128) is read and written once, next
// to which a few tokens are nothing. Output columns are independent, so a block takes 32 columns of
// one head: 4 blocks a head at dv = 128, each with 16 KB of the state in registers (32 a thread) and
// no exchange with any other block. Thread (rg, cg) owns rows 8 rg .. 8 rg + 7 and columns
// 4 cg .. 4 cg + 3, so that 8 lanes read a whole 128-byte row segment with 16-byte loads, all 8 of a
// thread in flight together. The sum over rows runs through two shuffles and, once for all tokens,
// shared memory.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fla {

struct DecodeTensor {
  const void* ptr;
  long long sb, sh, sn;  // element strides; innermost stride 1
};

struct DecodeParams {
  DecodeTensor q, k, v, o;
  const float* s_init;  // [bh][dk][dv] or null; may be the same array as s_final
  float* s_final;       // same shape, or null
  int heads, tokens, dk, dv;
};

constexpr int kDecodeThreads = 128;
constexpr int kDecodeCols = 32;       // columns of the state per block
constexpr int kDecodeRows = 128;      // rows a block covers: 16 groups of 8
constexpr int kDecodeMaxTokens = 16;  // longest call the kernel has room for, see use_decode()

template <bool HALF>
__device__ __forceinline__ float decode_load(const void* base, long long idx) {
  return HALF ? __half2float(static_cast<const __half*>(base)[idx])
              : __bfloat162float(static_cast<const __nv_bfloat16*>(base)[idx]);
}

template <bool HALF>
__global__ void __launch_bounds__(kDecodeThreads)
fla_decode_kernel(const DecodeParams p) {
  __shared__ float sq[kDecodeMaxTokens][kDecodeRows];
  __shared__ float sk[kDecodeMaxTokens][kDecodeRows];
  __shared__ float sv[kDecodeMaxTokens][kDecodeCols];
  __shared__ float part[kDecodeMaxTokens][4][kDecodeCols];  // per warp: sum over its 32 rows
  const int bh = blockIdx.y;
  const int b = bh / p.heads, h = bh % p.heads;
  const int col0 = blockIdx.x * kDecodeCols;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cg = tid & 7, row0 = (tid >> 3) * 8;
  const int c = col0 + cg * 4;
  const size_t base = static_cast<size_t>(bh) * p.dk * p.dv;
  // rows of dv floats are 16-byte aligned when dv % 4 == 0 (the state arrays themselves are checked
  // by the caller of the kernel)
  const bool vec = (p.dv & 3) == 0 && c + 4 <= p.dv;
  float s[8][4];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[r][j] = 0.f;
  if (p.s_init != nullptr) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int row = row0 + r;
      if (row < p.dk) {
        const float* src = p.s_init + base + static_cast<size_t>(row) * p.dv + c;
        if (vec) {
          const float4 x = *reinterpret_cast<const float4*>(src);
          s[r][0] = x.x; s[r][1] = x.y; s[r][2] = x.z; s[r][3] = x.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (c + j < p.dv) s[r][j] = src[j];
        }
      }
    }
  }
  // the tokens' rows as fp32; rows and columns outside the head dims count as zero
  const long long qo = b * p.q.sb + h * p.q.sh, ko = b * p.k.sb + h * p.k.sh, vo = b * p.v.sb + h * p.v.sh;
  for (int t = 0; t < p.tokens; ++t) {
    sq[t][tid] = tid < p.dk ? decode_load<HALF>(p.q.ptr, qo + t * p.q.sn + tid) : 0.f;
    sk[t][tid] = tid < p.dk ? decode_load<HALF>(p.k.ptr, ko + t * p.k.sn + tid) : 0.f;
    if (tid < kDecodeCols)
      sv[t][tid] = col0 + tid < p.dv ? decode_load<HALF>(p.v.ptr, vo + t * p.v.sn + col0 + tid) : 0.f;
  }
  __syncthreads();
#pragma unroll 1
  for (int t = 0; t < p.tokens; ++t) {
    const float4 v4 = *reinterpret_cast<const float4*>(&sv[t][cg * 4]);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float kr = sk[t][row0 + r], qr = sq[t][row0 + r];
      s[r][0] += kr * v4.x; s[r][1] += kr * v4.y; s[r][2] += kr * v4.z; s[r][3] += kr * v4.w;
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j] += qr * s[r][j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // the warp's four row groups
      acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 8);
      acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 16);
    }
    if (lane < 8) *reinterpret_cast<float4*>(&part[t][warp][cg * 4]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  }
  if (p.s_final != nullptr) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int row = row0 + r;
      if (row < p.dk) {
        float* dst = p.s_final + base + static_cast<size_t>(row) * p.dv + c;
        if (vec) {
          *reinterpret_cast<float4*>(dst) = make_float4(s[r][0], s[r][1], s[r][2], s[r][3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (c + j < p.dv) dst[j] = s[r][j];
        }
      }
    }
  }
  __syncthreads();
  for (int idx = tid; idx < p.tokens * kDecodeCols; idx += kDecodeThreads) {
    const int t = idx / kDecodeCols, cc = idx % kDecodeCols;
    if (col0 + cc < p.dv) {
      const float x = (part[t][0][cc] + part[t][1][cc]) + (part[t][2][cc] + part[t][3][cc]);
      const long long at = b * p.o.sb + h * p.o.sh + t * p.o.sn + col0 + cc;
      if (HALF) static_cast<__half*>(const_cast<void*>(p.o.ptr))[at] = __float2half_rn(x);
      else static_cast<__nv_bfloat16*>(const_cast<void*>(p.o.ptr))[at] = __float2bfloat16_rn(x);
    }
  }
}

}  // namespace fla
