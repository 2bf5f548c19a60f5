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
//
// Several tokens (MULTI) take the same sums in another order,
//     o_t = q_t S_0 + sum_{j <= t} (q_t . k_j) v_j,   S = S_0 + sum_t k_t^T v_t:
// the state stays what it was until the end and is then rounded once a call, like the tensor cores'
// sum, and not once a token (fp16, 8 tokens from a state of 256: 6.9e-8 off the exact state token by token,
// 2.7e-8 this way), and no token waits for the one before. Seven blocks have to fit an SM (72
// registers), or the 1024 blocks of 256 heads take a second round. 128 x 128, token by token and this way:
// 256 heads, 2 tokens 8.2 and 9.7 us, 16 tokens 20.3 and 22.5; 16 heads, 16 tokens 10.9 and 10.8.
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
// floats from one token's q or k row to the next in shared memory: 8 banks on, so that the eight rows
// of a score fragment, two words a lane, touch different banks
constexpr int kDecodeStride = kDecodeRows + 8;

template <bool HALF>
__device__ __forceinline__ float decode_load(const void* base, long long idx) {
  return HALF ? __half2float(static_cast<const __half*>(base)[idx])
              : __bfloat162float(static_cast<const __nv_bfloat16*>(base)[idx]);
}

template <bool HALF>
__device__ __forceinline__ uint32_t decode_pair(const float* src) {
  const float2 x = *reinterpret_cast<const float2*>(src);
  if (HALF) {
    const __half2 h = __floats2half2_rn(x.x, x.y);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  const __nv_bfloat162 h = __floats2bfloat162_rn(x.x, x.y);
  return *reinterpret_cast<const uint32_t*>(&h);
}

template <bool HALF>
__device__ __forceinline__ void decode_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                           uint32_t b0, uint32_t b1) {
  if (HALF)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <bool HALF, bool MULTI>
__global__ void __launch_bounds__(kDecodeThreads, 7)
fla_decode_kernel(const DecodeParams p) {
  constexpr int kTokens = MULTI ? kDecodeMaxTokens : 1;
  __shared__ __align__(16) float sq[kTokens][kDecodeStride];
  __shared__ __align__(16) float sk[kTokens][kDecodeStride];
  __shared__ __align__(16) float sv[kTokens][kDecodeCols];
  __shared__ __align__(16) float part[kTokens][4][kDecodeCols];  // per warp: sum over its 32 rows
  __shared__ __align__(16) float score[kTokens][kTokens];        // q_t . k_j
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
  // the tokens' rows as fp32; rows and columns outside the head dims count as zero. Four tokens' loads
  // are in flight together: one after the other they were most of the time a token took (0.5 us).
  const long long qo = b * p.q.sb + h * p.q.sh, ko = b * p.k.sb + h * p.k.sh, vo = b * p.v.sb + h * p.v.sh;
  const int tokens = MULTI ? p.tokens : 1;
  constexpr int kBatch = MULTI ? 4 : 1;
  const bool has_v = tid < kDecodeCols && col0 + tid < p.dv;
#pragma unroll 1
  for (int t0 = 0; t0 < tokens; t0 += kBatch) {
    float xq[kBatch], xk[kBatch], xv[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int t = t0 + i;
      if (t >= tokens) break;
      xq[i] = xk[i] = xv[i] = 0.f;
      if (tid < p.dk) {
        xq[i] = decode_load<HALF>(p.q.ptr, qo + t * p.q.sn + tid);
        xk[i] = decode_load<HALF>(p.k.ptr, ko + t * p.k.sn + tid);
      }
      if (has_v) xv[i] = decode_load<HALF>(p.v.ptr, vo + t * p.v.sn + col0 + tid);
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      if (t0 + i >= tokens) break;
      sq[t0 + i][tid] = xq[i];
      sk[t0 + i][tid] = xk[i];
      if (tid < kDecodeCols) sv[t0 + i][tid] = xv[i];
    }
  }
  __syncthreads();
  if (MULTI) {
    // Scores, while the state is still on its way. Up to four tokens: one warp a token, sums through
    // shuffles. More: a 16 x 16 tile over 128 columns,
    // far below one tcgen05 tile, as two 16 x 8 mma.sync tiles (the operands go back to the 16 bits they
    // came in). That chain takes about 1 us, too much for a few tokens, and the shuffles of 16 tokens
    // take twice that. Rows and columns of tokens that do not exist hold anything and are not read.
    // Neighbouring blocks give the tiles to different warps, i.e. to different quarters of the SM.
    const int half = (warp + blockIdx.x + blockIdx.y) & 3;
    if (tokens <= 4) {
      if (warp < tokens) {
        const float4 q4 = *reinterpret_cast<const float4*>(&sq[warp][lane * 4]);
#pragma unroll 1
        for (int j = 0; j <= warp; ++j) {
          const float4 k4 = *reinterpret_cast<const float4*>(&sk[j][lane * 4]);
          float x = (q4.x * k4.x + q4.y * k4.y) + (q4.z * k4.z + q4.w * k4.w);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
          if (lane == 0) score[warp][j] = x;
        }
      }
    } else if (half < 2 && half * 8 < tokens) {
      const int g = lane >> 2, pr = (lane & 3) * 2;
      float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
      for (int k0 = 0; k0 < kDecodeRows; k0 += 16) {
        const uint32_t a0 = decode_pair<HALF>(&sq[g][k0 + pr]), a1 = decode_pair<HALF>(&sq[g + 8][k0 + pr]);
        const uint32_t a2 = decode_pair<HALF>(&sq[g][k0 + 8 + pr]), a3 = decode_pair<HALF>(&sq[g + 8][k0 + 8 + pr]);
        const uint32_t b0 = decode_pair<HALF>(&sk[half * 8 + g][k0 + pr]);
        const uint32_t b1 = decode_pair<HALF>(&sk[half * 8 + g][k0 + 8 + pr]);
        decode_mma<HALF>(d, a0, a1, a2, a3, b0, b1);
      }
      *reinterpret_cast<float2*>(&score[g][half * 8 + pr]) = make_float2(d[0], d[1]);
      *reinterpret_cast<float2*>(&score[g + 8][half * 8 + pr]) = make_float2(d[2], d[3]);
    }
  } else {
    const float4 v4 = *reinterpret_cast<const float4*>(&sv[0][cg * 4]);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float kr = sk[0][row0 + r];
      s[r][0] += kr * v4.x; s[r][1] += kr * v4.y; s[r][2] += kr * v4.z; s[r][3] += kr * v4.w;
    }
  }
#pragma unroll 1
  for (int t = 0; t < tokens; ++t) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int rr = 0; rr < 8; rr += 4) {
      const float4 q4 = *reinterpret_cast<const float4*>(&sq[t][row0 + rr]);
      const float qr[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j] += qr[i] * s[rr + i][j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // the warp's four row groups
      acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 8);
      acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 16);
    }
    if (lane < 8) *reinterpret_cast<float4*>(&part[t][warp][cg * 4]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  }
  if (MULTI) {
    // what the tokens add to the state, four of the thread's rows at a time
    if (p.s_final != nullptr) {
#pragma unroll
      for (int rr = 0; rr < 8; rr += 4) {
        float add[4][4];
        {
          const float4 v4 = *reinterpret_cast<const float4*>(&sv[0][cg * 4]);
          const float4 k4 = *reinterpret_cast<const float4*>(&sk[0][row0 + rr]);
          const float kr[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            add[i][0] = kr[i] * v4.x; add[i][1] = kr[i] * v4.y;
            add[i][2] = kr[i] * v4.z; add[i][3] = kr[i] * v4.w;
          }
        }
#pragma unroll 1
        for (int t = 1; t < tokens; ++t) {
          const float4 v4 = *reinterpret_cast<const float4*>(&sv[t][cg * 4]);
          const float4 k4 = *reinterpret_cast<const float4*>(&sk[t][row0 + rr]);
          const float kr[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            add[i][0] += kr[i] * v4.x; add[i][1] += kr[i] * v4.y;
            add[i][2] += kr[i] * v4.z; add[i][3] += kr[i] * v4.w;
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) s[rr + i][j] += add[i][j];
      }
    }
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
  // a thread takes four columns of one token
  const int t = tid >> 3, cc = (tid & 7) * 4;
  if (t < tokens && col0 + cc < p.dv) {
    float x[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float4 y = *reinterpret_cast<const float4*>(&part[t][w][cc]);
      x[0] += y.x; x[1] += y.y; x[2] += y.z; x[3] += y.w;
    }
    if (MULTI) {
#pragma unroll 1
      for (int j = 0; j <= t; ++j) {
        const float sc = score[t][j];
        const float4 y = *reinterpret_cast<const float4*>(&sv[j][cc]);
        x[0] += sc * y.x; x[1] += sc * y.y; x[2] += sc * y.z; x[3] += sc * y.w;
      }
    }
    const long long at = b * p.o.sb + h * p.o.sh + t * p.o.sn + col0 + cc;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (col0 + cc + j >= p.dv) break;
      if (HALF) static_cast<__half*>(const_cast<void*>(p.o.ptr))[at + j] = __float2half_rn(x[j]);
      else static_cast<__nv_bfloat16*>(const_cast<void*>(p.o.ptr))[at + j] = __float2bfloat16_rn(x[j]);
    }
  }
}

}  // namespace fla
