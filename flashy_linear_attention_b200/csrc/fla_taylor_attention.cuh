// Causal linear attention on second-order Taylor features of raw q, k (d = 8 or 16), the features formed on
// chip, for sm_100a:   out_i = sum_{j<=i} f(s_ij) v_j,  f(s) = 1 + s + s^2 / 2,  s_ij = q_i . k_j / sqrt(d).
//
// fla_taylor.cuh writes the 1 + d + d^2 features (273 at d = 16) to HBM for the SmallVHD kernels: 2.2 KB a
// token and pass against the 320 bytes that q, k, v and the output have. Here a CTA reads the raw rows and
// forms the features it needs in shared memory, once per unordered pair of columns,
//     phi(x) = [x_a (16 columns), x_a x_b for a <= b, 1]                     160 columns at d = 16, 64 at 8
// with the weights of the expansion (1 / sqrt(d), 1 / d or 1 / 2d, 1) on the state side, where they are
// applied in fp32:  phi(q) . W phi(k) = f(s). Inside a chunk the scores come from the raw columns alone,
// s in one MMA step of 16 columns, and f is evaluated in fp32.
//
// One loop serves three roles. Rows x and columns y are the raw tensors, Z = sum b^T phi(y) the state:
//     forward   x = q, y = k, b = v            out = f(s) b + phi(x) W Z
//     dQ        x = q, y = k, a = dO, b = v    dx  = T y + J(x) (a W Z^T)     T = (a b^T) f'(s) / sqrt(d)
//     dK, dV    x = k, y = q, a = v, b = dO    both, from the last chunk to the first
// J(x) is the transposed Jacobian of phi: the gradient of phi's 160 columns stays fp32 in tensor memory, where
// the output warps contract it with the row's x. T is rounded to 16 bits as an MMA operand.
//
// Bound by the instructions of the warps around the tensor core, not by HBM (a chunk's 40 - 80 KB take 900 -
// 1600 cycles) or the MMAs (1700 - 2700): a chunk takes 3000 cycles forward and 5000 for dK and dV. So the
// feature products and the polynomial are packed operations on pairs, diagonal masks are applied to the packed result, and
// the roles' code is kept short: they all run at once and share the instruction cache (with the MMA loops and the
// conversions unrolled per mask the same work took 42 and 144 us instead of 32 and 96).
// 128 heads x 2048 tokens, d = 16, 64 value columns: forward 32 us and backward 96, against 130 and 355 through
// features in memory; relative error against 64 bits 2.3e-3 (out), 2.6e-3 (dq, dk), there 2.4e-3 and 3.1e-3.
// (Counters: issue slots 39 % and 33 % busy, tensor pipe 38 % and 32 % of active cycles, DRAM 20 % and 13 %.) A head has one
// CTA, resp. two, whatever its length: few heads leave SMs idle, at d = 16 with less time all the same (1 head x 8192:
// 103 + 174 us against 240 + 353), at d = 8 not, see the caller's rule.
//
// CTA layout (576 threads, one CTA per SM):
//   warp 0        TMA producer: a and b tiles, two stages
//   warp 1        MMA issuer (one elected lane) and TMEM owner
//   warps 2-9     converters: scores -> f(s) and T in 16 bits (TMEM), state -> 16 bits (shared memory)
//   warps 10-13   outputs: contraction to dx, accumulator -> 16 bits -> staging -> TMA store
//   warps 14-17   feature generators, a token row per thread
#pragma once
#include "fla_kernel.cuh"

namespace fla {

struct RawRows {  // [B, H, N, d] bf16, unit innermost stride, rows 16-byte aligned
  const __nv_bfloat16* ptr;
  long long sb, sh, sn;
};
struct TaylorProblem {
  CUtensorMap a, b;  // box 64 x 128
  CUtensorMap o;     // box 64 x 32
  RawRows x, y, dx;
  int flags;         // kFlagDescending | kFlagUpperMask for dK, dV
  int want_o, want_dx;
};
struct TaylorParams {
  TaylorProblem prob[2];
  int heads, nchunks, n_tokens;
  int* status;       // see KernelParams
  unsigned wait_limit_us;
  int debug_withhold;
};

constexpr int kTaylorThreads = 576;

template <int D>
struct TaylorCfg {
  static constexpr int PAIRS = D * (D + 1) / 2;
  static constexpr int NF = (16 + PAIRS + 1 + 15) / 16 * 16;  // feature columns
  static constexpr int GROUPS = (NF + 63) / 64;
  static constexpr int PHI_BYTES = GROUPS * kGroupBytes;
  static constexpr int ZB_GROUP = 64 * 128;  // 64 rows of a 64-column group
  // The raw rows of y and x of two chunks are the four 16-column quarters of one group: y, x, y', x'.
  static constexpr int RAW_OFF = 0, Y_OFF = kGroupBytes, X_OFF = Y_OFF + PHI_BYTES;
  static constexpr int B_OFF = X_OFF + PHI_BYTES, A_OFF = B_OFF + 2 * kGroupBytes;
  static constexpr int ZB_OFF = A_OFF + 2 * kGroupBytes, OST_OFF = ZB_OFF + GROUPS * ZB_GROUP;
  static constexpr int BAR_OFF = OST_OFF + kGroupBytes;
  static constexpr int SMEM_BYTES = 1024 + BAR_OFF + 256;
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
  // tensor memory columns: state, scores (then the gradient of phi(x)), a b^T (then T and T y), output
  static constexpr int Z_COL = 0, P_COL = 160, T_COL = 320, O_COL = 448, TY_COL = T_COL + 32;
  static_assert(NF <= 160, "tensor memory budget");
  // The quadratic columns come in 16-bit pairs, one packed product each: word w of them is
  //     x_a (x_2m, x_2m+1), m from (a + 1) / 2 on, for a = 0, 1, ...     then (x_a^2, x_a+2^2) for a = 1, 5, ...
  static constexpr int WORDS = PAIRS / 2, DIAG = WORDS - D / 4;  // first word of the squares left over
  __host__ __device__ static constexpr int word_a(int w) {
    if (w >= DIAG) return 4 * (w - DIAG) + 1;
    int a = 0;
    while (w >= D / 2 - (a + 1) / 2) { w -= D / 2 - (a + 1) / 2; ++a; }
    return a;
  }
  __host__ __device__ static constexpr int word_m(int w) {
    int a = 0;
    while (w >= D / 2 - (a + 1) / 2) { w -= D / 2 - (a + 1) / 2; ++a; }
    return (a + 1) / 2 + w;
  }
  __host__ __device__ static constexpr bool square(int idx) {  // column 16 + idx
    const int w = idx / 2;
    return w >= DIAG || word_a(w) == 2 * word_m(w) + idx % 2;
  }
  static constexpr float kLinear = D == 16 ? 0.25f : 0.35355339059327379f;  // 1 / sqrt(d)
  __host__ __device__ static constexpr float weight(int f) {
    return f < 16 ? kLinear
                  : f < 16 + PAIRS ? (square(f - 16) ? 0.5f / D : 1.f / D) : f == 16 + PAIRS ? 1.f : 0.f;
  }
};

// Two fp32 values in one register pair: a packed FMA or multiplication takes one issue slot for both.
__device__ __forceinline__ unsigned long long pair_of(float lo, float hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ unsigned long long pair_of(uint32_t lo, uint32_t hi) {
  return pair_of(__uint_as_float(lo), __uint_as_float(hi));
}
__device__ __forceinline__ float2 unpair(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// Products of bf16 pairs: exact, then rounded once, like an fp32 product that is rounded to bf16.
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

template <int D>
__global__ void __launch_bounds__(kTaylorThreads, 1)
fla_taylor_attention_kernel(const __grid_constant__ TaylorParams p) {
  using cfg = TaylorCfg<D>;
  constexpr int NF = cfg::NF;
  extern __shared__ uint8_t smem_raw[];
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const TaylorProblem& pr = p.prob[blockIdx.x];
  const int bh = blockIdx.z;
  const int h = bh % p.heads, b = bh / p.heads;
  const bool want_o = pr.want_o != 0, want_dx = pr.want_dx != 0;
  const bool descending = (pr.flags & kFlagDescending) != 0, upper_flag = (pr.flags & kFlagUpperMask) != 0;
  const int n_iter = p.nchunks;
  auto mem_chunk = [&](int i) { return descending ? n_iter - 1 - i : i; };

  const uint32_t raw_addr = ptx::smem_u32(smem_raw);
  const uint32_t smem_base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - raw_addr);
  const uint32_t raw_tile = smem_base + cfg::RAW_OFF, y_addr = smem_base + cfg::Y_OFF, x_addr = smem_base + cfg::X_OFF;
  const uint32_t zb_addr = smem_base + cfg::ZB_OFF, ost_addr = smem_base + cfg::OST_OFF;
  auto b_tile = [&](int i) { return smem_base + cfg::B_OFF + (i & 1) * kGroupBytes; };
  auto a_tile = [&](int i) { return smem_base + cfg::A_OFF + (i & 1) * kGroupBytes; };
  auto bar = [&](int i) { return smem_base + cfg::BAR_OFF + 8u * i; };
  auto full_bar = [&](int i) { return bar(i & 1); };        // a and b tiles of chunk i have arrived
  auto empty_bar = [&](int i) { return bar(2 + (i & 1)); };
  const uint32_t y_ready = bar(4);    // features of y and both raw rows written (128 arrivals)
  const uint32_t y_free = bar(5);
  const uint32_t p_full = bar(6);     // scores (and a b^T) complete
  const uint32_t pb_ready = bar(7);   // and converted (256)
  const uint32_t z_full = bar(8);     // state complete, its copy no longer read
  const uint32_t zb_ready = bar(9);   // copy written (256)
  const uint32_t o_full = bar(10), o_free = bar(11);    // accumulator (128)
  const uint32_t dx_full = bar(12), dx_free = bar(13);  // gradient of phi(x), and T y (128)
  const uint32_t drained = bar(14);
  const uint32_t x_ready = bar(15), x_free = bar(16);  // features of x (128; want_o)
  volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(smem_gen + cfg::BAR_OFF + 17 * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + cfg::BAR_OFF + 17 * 8 + 4);

  if (threadIdx.x == 0) {
    abort_flag[0] = 0;
    abort_flag[1] = static_cast<int>(p.wait_limit_us);
    for (int i = 0; i < 4; ++i) ptx::mbar_init(bar(i), 1);
    ptx::mbar_init(y_ready, 128);
    ptx::mbar_init(y_free, 1);
    ptx::mbar_init(x_ready, 128);
    ptx::mbar_init(x_free, 1);
    ptx::mbar_init(p_full, 1);
    ptx::mbar_init(pb_ready, 256);
    ptx::mbar_init(z_full, 1);
    ptx::mbar_init(zb_ready, 256);
    ptx::mbar_init(o_full, 1);
    ptx::mbar_init(o_free, 128);
    ptx::mbar_init(dx_full, 1);
    ptx::mbar_init(dx_free, 128);
    ptx::mbar_init(drained, 1);
    ptx::fence_barrier_init();
    ptx::fence_proxy_async_smem();
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_holder)), 512);
    ptx::tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    if (want_dx) ptx::prefetch_tensormap(&pr.a);
    ptx::prefetch_tensormap(&pr.b);
    if (want_o) ptx::prefetch_tensormap(&pr.o);
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_holder, 0);  // provably warp-uniform
  auto wait_uniform = [&](uint32_t bar_addr, uint32_t parity) {
    const int ok = ptx::mbar_wait(bar_addr, parity, abort_flag) ? 1 : 0;
    return __all_sync(0xffffffffu, ok) != 0;
  };
  auto wait_tmem = [&](uint32_t bar_addr, uint32_t parity) {
    const bool up = wait_uniform(bar_addr, parity);
    if (up) ptx::tc_fence_after();
    return up;
  };
  auto load_row = [&](const RawRows& t, int tok, uint32_t (&w)[D / 2]) {
#pragma unroll
    for (int j = 0; j < D / 8; ++j) {
      uint4 x = make_uint4(0u, 0u, 0u, 0u);
      if (tok < p.n_tokens) x = __ldg(reinterpret_cast<const uint4*>(t.ptr + b * t.sb + h * t.sh + tok * t.sn) + j);
      w[4 * j] = x.x; w[4 * j + 1] = x.y; w[4 * j + 2] = x.z; w[4 * j + 3] = x.w;
    }
  };
  bool issuer = false;

  if (warp == 0) {
    // ================================================================ TMA producer
    const bool leader = ptx::elect_one();
    for (int i = 0; i < n_iter; ++i) {
      if (!wait_uniform(empty_bar(i), ((i >> 1) & 1) ^ 1u)) break;
      if (leader) {
        const int tok = mem_chunk(i) * kChunk;
        ptx::mbar_expect_tx(full_bar(i), (want_dx ? 2 : 1) * kGroupBytes);
        if (!(p.debug_withhold && i == 0)) ptx::tma_load_4d(b_tile(i), &pr.b, full_bar(i), 0, tok, h, b);
        if (want_dx) ptx::tma_load_4d(a_tile(i), &pr.a, full_bar(i), 0, tok, h, b);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    // ================================================================ MMA issuer
    constexpr uint32_t IDESC_P = ptx::make_idesc(128, 128, false, false);  // x y^T, a b^T
    constexpr uint32_t IDESC_XZ = ptx::make_idesc(128, 64, false, false);  // phi(x) Z^T: contracts Z's columns
    constexpr uint32_t IDESC_Z = ptx::make_idesc(128, NF, true, true);     // Z += b^T phi(y)
    constexpr uint32_t IDESC_PB = ptx::make_idesc(128, 64, false, true);   // f(s) b
    constexpr uint32_t IDESC_TY = ptx::make_idesc(128, 16, false, true);   // T y
    constexpr uint32_t IDESC_AZ = ptx::make_idesc(128, NF, false, true);   // a Z: contracts Z's rows
    const uint32_t tZ = tmem_base + cfg::Z_COL, tP = tmem_base + cfg::P_COL, tT = tmem_base + cfg::T_COL;
    const uint32_t tO = tmem_base + cfg::O_COL, tTy = tmem_base + cfg::TY_COL;
    const bool leader = ptx::elect_one();
    issuer = leader;
    const uint32_t x_k = ptx::desc_lo(x_addr, 16), y_mn = ptx::desc_lo(y_addr, kGroupBytes);
    const uint32_t raw_k = ptx::desc_lo(raw_tile, 16), raw_mn = ptx::desc_lo(raw_tile, kGroupBytes);
    const uint32_t zb_k = ptx::desc_lo(zb_addr, 16), zb_mn = ptx::desc_lo(zb_addr, cfg::ZB_GROUP);
    auto k_step = [](int kk, int group) { return static_cast<uint32_t>(((kk >> 2) * group + (kk & 3) * 32) >> 4); };
    auto half_step = [](int kk) { return static_cast<uint32_t>((kk >> 2) * 64 + (kk & 3) * 8); };  // 16-bit tile, in two halves
    for (int i = 0; i < n_iter; ++i) {
      const bool last = i + 1 == n_iter, have_z = i > 0;
      const uint32_t b_k = ptx::desc_lo(b_tile(i), 16), b_mn = ptx::desc_lo(b_tile(i), kGroupBytes);
      const uint32_t a_k = ptx::desc_lo(a_tile(i), 16);
      const uint32_t raw_y = (i & 1) * (64 >> 4), raw_x = raw_y + (32 >> 4);  // this chunk's quarters
      if (!wait_uniform(y_ready, i & 1)) break;
      if (!wait_uniform(full_bar(i), (i >> 1) & 1)) break;
      if (want_dx && have_z && !wait_uniform(dx_free, (i - 1) & 1)) break;  // the score tile's place is free
      ptx::tc_fence_after();
      {
        ptx::mma_ss_on(leader, tP, raw_k + raw_x, raw_k + raw_y, ptx::kDescHi, IDESC_P, 0u);
        if (want_dx) {
#pragma unroll 1
          for (int kk = 0; kk < 4; ++kk)
            ptx::mma_ss_on(leader, tT, a_k + k_step(kk, 0), b_k + k_step(kk, 0), ptx::kDescHi, IDESC_P, kk > 0 ? 1u : 0u);
        }
        ptx::tc_commit_on(leader, p_full);
      }
      // Z += b^T phi(y); the previous Z has been converted
      if (have_z && !wait_tmem(zb_ready, (i - 1) & 1)) break;
      if (!last) {
        // The instruction spans 128 rows of Z; the upper 64 read what follows the b tile in shared memory
        // and land in tensor-memory lanes nobody reads.
#pragma unroll 1
        for (int kk = 0; kk < kChunk / 16; ++kk)
          ptx::mma_ss_on(leader, tZ, b_mn + kk * (2048 >> 4), y_mn + kk * (2048 >> 4), ptx::kDescHi, IDESC_Z, (have_z || kk > 0) ? 1u : 0u);
        ptx::tc_commit_on(leader, y_free);
      }
      if (want_o) {
        if (!wait_uniform(x_ready, i & 1)) break;
        if (have_z) {
          if (!wait_tmem(o_free, (i - 1) & 1)) break;
#pragma unroll 1
          for (int kk = 0; kk < NF / 16; ++kk)
            ptx::mma_ss_on(leader, tO, x_k + k_step(kk, kGroupBytes), zb_k + k_step(kk, cfg::ZB_GROUP), ptx::kDescHi, IDESC_XZ, kk > 0 ? 1u : 0u);
        }
        if (!last) ptx::tc_commit_on(leader, x_free);
      }
      if (!last && !want_dx) ptx::tc_commit_on(leader, z_full);
      if (!wait_tmem(pb_ready, i & 1)) break;
      {
        if (want_o) {
#pragma unroll 1
          for (int kk = 0; kk < kChunk / 16; ++kk)
            ptx::mma_ts_on(leader, tO, tP + half_step(kk), b_mn + kk * (2048 >> 4), ptx::kDescHi, IDESC_PB, (have_z || kk > 0) ? 1u : 0u);
          ptx::tc_commit_on(leader, o_full);
        }
        if (want_dx) {
          if (have_z) {  // into the place of the scores, which the conversion and f(s) b have used up
#pragma unroll 1
            for (int kk = 0; kk < 4; ++kk)
              ptx::mma_ss_on(leader, tP, a_k + k_step(kk, 0), zb_mn + kk * (2048 >> 4), ptx::kDescHi, IDESC_AZ, kk > 0 ? 1u : 0u);
          }
#pragma unroll 1
          for (int kk = 0; kk < kChunk / 16; ++kk)
            ptx::mma_ts_on(leader, tTy, tT + half_step(kk), raw_mn + raw_y + kk * (2048 >> 4), ptx::kDescHi, IDESC_TY, kk > 0 ? 1u : 0u);
          ptx::tc_commit_on(leader, dx_full);
          if (!last) ptx::tc_commit_on(leader, z_full);
        }
        ptx::tc_commit_on(leader, empty_bar(i));
      }
      __syncwarp();
    }
  } else if (warp < 10) {
    // ================================================================ converters
    const int half = (warp - 2) >> 2;
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    constexpr float cs = cfg::kLinear;
    uint32_t rs[32], rt[32], pk[16];
    for (int i = 0; i < n_iter; ++i) {
      if (!wait_tmem(p_full, i & 1)) break;
      // This group's 64 columns in two blocks of 32; the 16-bit forms go into the first half of the
      // group's own fp32 columns, which are read by then.
      // f = ((1 + s)^2 + 1) / 2,  T = (a b^T) (1 + s) / sqrt(d): two packed operations each for two scores
      auto convert = [&](auto scores_c, uint32_t dst, bool diagonal) {
        constexpr bool kScores = decltype(scores_c)::value;
        constexpr float kRoot = 0.70710678118654752f;
        constexpr float k1 = kScores ? cs * kRoot : cs * cs, k0 = kScores ? kRoot : cs;
        const unsigned long long m1 = pair_of(k1, k1), m0 = pair_of(k0, k0), half2 = pair_of(0.5f, 0.5f);
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const unsigned long long u = fma2(pair_of(rs[2 * c], rs[2 * c + 1]), m1, m0);
          const float2 v = unpair(kScores ? fma2(u, u, half2) : mul2(u, pair_of(rt[2 * c], rt[2 * c + 1])));
          pk[c] = ptx::pack_bf16x2(v.x, v.y);
        }
        if (diagonal) {
          // columns up to the row are kept, or (upper) all but those before it
          const int edge = upper_flag ? lane - 1 : lane;
          const uint32_t flip = upper_flag ? 0xffffffffu : 0u;
#pragma unroll
          for (int c = 0; c < 16; ++c) pk[c] &= (edge > 2 * c ? 0xffffffffu : edge == 2 * c ? 0x0000ffffu : 0u) ^ flip;
        }
        ptx::tmem_st16(dst, pk);
      };
#pragma unroll 1
      for (int j = 0; j < 2; ++j) {
        const int cb = half * 2 + j;
        const bool masked = upper_flag ? cb < quad : cb > quad;  // warp-uniform
        const uint32_t src_s = lane_base + cfg::P_COL + cb * 32, src_t = lane_base + cfg::T_COL + cb * 32;
        const uint32_t dst_s = lane_base + cfg::P_COL + half * 64 + j * 16, dst_t = lane_base + cfg::T_COL + half * 64 + j * 16;
        if (masked) {
#pragma unroll
          for (int c = 0; c < 16; ++c) pk[c] = 0u;
          if (want_o) ptx::tmem_st16(dst_s, pk);
          if (want_dx) ptx::tmem_st16(dst_t, pk);
          continue;
        }
        if (want_dx) ptx::tmem_ld32x2(src_s, rs, src_t, rt);
        else ptx::tmem_ld32(src_s, rs);
        if (want_o) convert(std::true_type{}, dst_s, cb == quad);
        if (want_dx) convert(std::false_type{}, dst_t, cb == quad);
      }
      ptx::tc_wait_st();
      ptx::tc_fence_before();
      ptx::mbar_arrive(pb_ready);
      if (i + 1 < n_iter) {
        // State -> weighted 16-bit copy, [64-column group][64 rows][128 B], 16-byte pieces XOR-swizzled by
        // (row % 8). The state has 64 rows: the lower two lane quadrants; the halves share its columns.
        if (!wait_tmem(z_full, i & 1)) break;
        if (quad < 2) {
          constexpr int kBlocks = NF / 32, kFirst = (kBlocks + 1) / 2;
          auto convert_block = [&](auto cb_c) {
            constexpr int CB = decltype(cb_c)::value;
            ptx::tmem_ld32(lane_base + cfg::Z_COL + CB * 32, rs);
            ptx::static_for<4>([&](auto jj) {
              constexpr int J = decltype(jj)::value, F = CB * 32 + J * 8;
              uint32_t w[4];
              ptx::static_for<4>([&](auto c) {
                constexpr int C = decltype(c)::value;
                constexpr float w0 = cfg::weight(F + 2 * C), w1 = cfg::weight(F + 2 * C + 1);
                w[C] = ptx::pack_bf16x2(w0 * __uint_as_float(rs[J * 8 + 2 * C]), w1 * __uint_as_float(rs[J * 8 + 2 * C + 1]));
              });
              ptx::st_shared_v4(zb_addr + (F >> 6) * cfg::ZB_GROUP + row * 128 + ((((F >> 3) & 7) ^ (row & 7)) << 4), w[0], w[1], w[2], w[3]);
            });
          };
          if (half == 0) ptx::static_for<kFirst>(convert_block);
          else ptx::static_for<kBlocks - kFirst>([&](auto c) { convert_block(std::integral_constant<int, decltype(c)::value + kFirst>{}); });
        }
        ptx::fence_proxy_async_smem();
        ptx::tc_fence_before();
        ptx::mbar_arrive(zb_ready);
      }
    }
  } else if (warp < 14) {
    // ================================================================ outputs
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t swz = static_cast<uint32_t>(row & 7);
    uint32_t ra[32], rb[32];
    for (int i = 0; i < n_iter; ++i) {
      const int tok = mem_chunk(i) * kChunk + row;
      if (want_dx) {
        uint32_t xw[D / 2];
        load_row(pr.x, tok, xw);
        unsigned long long acc[D / 2];  // dx in pairs
        if (!wait_tmem(dx_full, i & 1)) break;
        ptx::tmem_ld32(lane_base + cfg::TY_COL, ra);  // (16 columns of it)
#pragma unroll
        for (int m = 0; m < D / 2; ++m) acc[m] = pair_of(ra[2 * m], ra[2 * m + 1]);
        if (i > 0) {
          const unsigned long long ones = pair_of(1.f, 1.f);
          auto x_of = [&](int a) { return (a & 1) ? ptx::bf16_hi(xw[a >> 1]) : ptx::bf16_lo(xw[a >> 1]); };
          auto add_to = [&](int a, float v) {  // dx_a += v
            float2 f = unpair(acc[a >> 1]);
            ((a & 1) ? f.y : f.x) += v;
            acc[a >> 1] = pair_of(f.x, f.y);
          };
          unsigned long long row_sum = 0ull;  // of the words with one a, so far
          ptx::static_for<NF / 32>([&](auto cb_c) {
            constexpr int CB = decltype(cb_c)::value;
            ptx::tmem_ld32(lane_base + cfg::P_COL + CB * 32, ra);
            // the row is unpacked again for every block: unpacked it would not fit the registers
#pragma unroll
            for (int m = 0; m < D / 2; ++m) asm volatile("" : "+r"(xw[m]));
            ptx::static_for<16>([&](auto c) {
              constexpr int C = decltype(c)::value, F = CB * 32 + 2 * C, W = (F - 16) / 2;
              const unsigned long long gv = pair_of(ra[2 * C], ra[2 * C + 1]);
              if constexpr (F < D) {
                acc[F / 2] = fma2(gv, ones, acc[F / 2]);
              } else if constexpr (F >= 16 && W < cfg::DIAG) {
                constexpr int A = cfg::word_a(W), M = cfg::word_m(W);
                const float xa = x_of(A);
                acc[M] = fma2(gv, pair_of(xa, xa), acc[M]);
                row_sum = fma2(gv, pair_of(x_of(2 * M), x_of(2 * M + 1)), row_sum);
                if constexpr (M == D / 2 - 1) {
                  const float2 f = unpair(row_sum);
                  add_to(A, f.x + f.y);
                  row_sum = 0ull;
                }
              } else if constexpr (F >= 16 && W < cfg::WORDS) {
                constexpr int A = cfg::word_a(W);
                const float2 f = unpair(gv);
                add_to(A, 2.f * f.x * x_of(A));
                add_to(A + 2, 2.f * f.y * x_of(A + 2));
              }
            });
          });
        }
        if (tok < p.n_tokens) {
          uint4* dst = reinterpret_cast<uint4*>(const_cast<__nv_bfloat16*>(pr.dx.ptr) + b * pr.dx.sb + h * pr.dx.sh + tok * pr.dx.sn);
#pragma unroll
          for (int j = 0; j < D / 8; ++j) {
            uint32_t w[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float2 f = unpair(acc[4 * j + c]);
              w[c] = ptx::pack_bf16x2(f.x, f.y);
            }
            dst[j] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        ptx::tc_fence_before();
        ptx::mbar_arrive(dx_free);  // after the stores that consume what was loaded
      }
      if (want_o) {
        if (lane == 0) ptx::bulk_wait_group_read0();  // this warp's previous store has read its rows
        __syncwarp();
        if (!wait_tmem(o_full, i & 1)) break;
        ptx::tmem_ld32x2(lane_base + cfg::O_COL, ra, lane_base + cfg::O_COL + 32, rb);
        const uint32_t dst = ost_addr + row * 128;
        auto store_half = [&](uint32_t j0, const uint32_t (&r)[32]) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            ptx::st_shared_v4(dst + (((j0 + j) ^ swz) << 4),
                              ptx::pack_bf16x2(__uint_as_float(r[8 * j + 0]), __uint_as_float(r[8 * j + 1])),
                              ptx::pack_bf16x2(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3])),
                              ptx::pack_bf16x2(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5])),
                              ptx::pack_bf16x2(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7])));
        };
        store_half(0, ra);
        store_half(4, rb);
        ptx::tc_fence_before();
        ptx::mbar_arrive(o_free);
        ptx::fence_proxy_async_smem();
        __syncwarp();
        const int tok0 = mem_chunk(i) * kChunk + quad * 32;
        if (lane == 0 && tok0 < p.n_tokens) {
          ptx::tma_store_4d(&pr.o, ost_addr + quad * (32 * 128), 0, tok0, h, b);
          ptx::bulk_commit_group();
        }
      }
    }
    if (lane == 0) ptx::bulk_wait_group0();
  } else {
    // ================================================================ feature generators
    const int r = (warp - 14) * 32 + lane;
    const uint32_t swz = static_cast<uint32_t>(r & 7);
    uint32_t xv[D / 2], yv[D / 2];
    load_row(pr.y, mem_chunk(0) * kChunk + r, yv);
    load_row(pr.x, mem_chunk(0) * kChunk + r, xv);
    auto write_row = [&](uint32_t tile, const uint32_t (&v)[D / 2]) {
      ptx::static_for<NF / 8>([&](auto piece) {
        constexpr int P = decltype(piece)::value;
        uint32_t w[4];
        ptx::static_for<4>([&](auto c) {
          constexpr int WD = 4 * P + decltype(c)::value, W = WD - 8;  // word of the row, word of the products
          uint32_t& out = w[decltype(c)::value];
          if constexpr (WD < D / 2) {
            out = v[WD];
          } else if constexpr (W >= 0 && W < cfg::DIAG) {
            constexpr int A = cfg::word_a(W), M = cfg::word_m(W);
            out = mul_bf16x2(__byte_perm(v[A >> 1], 0u, (A & 1) ? 0x3232 : 0x1010), v[M]);
          } else if constexpr (W >= 0 && W < cfg::WORDS) {
            constexpr int A = cfg::word_a(W);
            const uint32_t x = __byte_perm(v[A >> 1], v[(A >> 1) + 1], 0x7632);  // (x_a, x_a+2), a odd
            out = mul_bf16x2(x, x);
          } else {
            out = W == cfg::WORDS ? 0x3F80u : 0u;  // the constant feature
          }
        });
        ptx::st_shared_v4(tile + (P >> 3) * kGroupBytes + r * 128 + (((P & 7) ^ swz) << 4), w[0], w[1], w[2], w[3]);
      });
    };
    auto write_raw = [&](int quarter, const uint32_t (&v)[D / 2]) {  // 16 columns: two pieces
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t dst = raw_tile + r * 128 + (((2 * quarter + j) ^ swz) << 4);
        if (j < D / 8) ptx::st_shared_v4(dst, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        else ptx::st_shared_v4(dst, 0u, 0u, 0u, 0u);
      }
    };
    for (int i = 0; i < n_iter; ++i) {
      // Z += b^T phi(y) of the chunk before is complete, and with it everything issued earlier: the last
      // readers of this chunk's quarters of the raw tile too
      bool up = i == 0 || wait_uniform(y_free, (i - 1) & 1);
      if (!up) break;
      write_raw((i & 1) * 2, yv);
      write_raw((i & 1) * 2 + 1, xv);
#pragma unroll 1
      for (int pass = 0; pass < (want_o ? 2 : 1); ++pass) {
        if (pass == 1 && i > 0) up = wait_uniform(x_free, (i - 1) & 1);
        if (!up) break;
        write_row(pass == 0 ? y_addr : x_addr, yv);
        ptx::fence_proxy_async_smem();
        ptx::mbar_arrive(pass == 0 ? y_ready : x_ready);
#pragma unroll
        for (int c = 0; c < D / 2; ++c) yv[c] = xv[c];
      }
      if (!up) break;
      if (i + 1 < n_iter) {
        load_row(pr.y, mem_chunk(i + 1) * kChunk + r, yv);
        load_row(pr.x, mem_chunk(i + 1) * kChunk + r, xv);
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  __syncwarp();
  if (warp == 1) {  // see fla_kernel.cuh
    if (issuer) ptx::tc_commit(drained);
    __syncwarp();
    wait_uniform(drained, 0);
  }
  if (*abort_flag) __nanosleep(100000);  // a wait gave up: let copies in flight land
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, 512);
  }
  if (threadIdx.x == 0 && *abort_flag && p.status != nullptr) atomicOr(p.status, 1);
}

}  // namespace fla
