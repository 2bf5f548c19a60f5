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
  static constexpr int Y_OFF = 0, X_OFF = PHI_BYTES, B_OFF = 2 * PHI_BYTES, A_OFF = B_OFF + 2 * kGroupBytes;
  static constexpr int ZB_OFF = A_OFF + 2 * kGroupBytes, OST_OFF = ZB_OFF + GROUPS * ZB_GROUP;
  static constexpr int BAR_OFF = OST_OFF + kGroupBytes;
  static constexpr int SMEM_BYTES = 1024 + BAR_OFF + 256;
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
  // tensor memory columns: state, scores (then the gradient of phi(x)), a b^T (then T and T y), output
  static constexpr int Z_COL = 0, P_COL = 160, T_COL = 320, O_COL = 448, TY_COL = T_COL + 32;
  static_assert(NF <= 160, "tensor memory budget");
  // first / second factor of column 16 + idx
  __host__ __device__ static constexpr int first(int idx) {
    int a = 0;
    while (idx >= D - a) idx -= D - a++;
    return a;
  }
  __host__ __device__ static constexpr int second(int idx) {
    int a = 0;
    while (idx >= D - a) idx -= D - a++;
    return a + idx;
  }
  static constexpr float kLinear = D == 16 ? 0.25f : 0.35355339059327379f;  // 1 / sqrt(d)
  __host__ __device__ static constexpr float weight(int f) {
    return f < 16 ? kLinear
                  : f < 16 + PAIRS ? (first(f - 16) == second(f - 16) ? 0.5f / D : 1.f / D) : f == 16 + PAIRS ? 1.f : 0.f;
  }
};

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
  const uint32_t y_addr = smem_base + cfg::Y_OFF, x_addr = smem_base + cfg::X_OFF;
  const uint32_t zb_addr = smem_base + cfg::ZB_OFF, ost_addr = smem_base + cfg::OST_OFF;
  auto b_tile = [&](int i) { return smem_base + cfg::B_OFF + (i & 1) * kGroupBytes; };
  auto a_tile = [&](int i) { return smem_base + cfg::A_OFF + (i & 1) * kGroupBytes; };
  auto bar = [&](int i) { return smem_base + cfg::BAR_OFF + 8u * i; };
  auto full_bar = [&](int i) { return bar(i & 1); };        // a and b tiles of chunk i have arrived
  auto empty_bar = [&](int i) { return bar(2 + (i & 1)); };
  const uint32_t phi_ready = bar(4);  // features of x and y written (128 arrivals)
  const uint32_t phi_free = bar(5);
  const uint32_t p_full = bar(6);     // scores (and a b^T) complete
  const uint32_t pb_ready = bar(7);   // and converted (256)
  const uint32_t z_full = bar(8);     // state complete, its copy no longer read
  const uint32_t zb_ready = bar(9);   // copy written (256)
  const uint32_t o_full = bar(10), o_free = bar(11);    // accumulator (128)
  const uint32_t dx_full = bar(12), dx_free = bar(13);  // gradient of phi(x), and T y (128)
  const uint32_t drained = bar(14);
  volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(smem_gen + cfg::BAR_OFF + 15 * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + cfg::BAR_OFF + 15 * 8 + 4);

  if (threadIdx.x == 0) {
    abort_flag[0] = 0;
    abort_flag[1] = static_cast<int>(p.wait_limit_us);
    for (int i = 0; i < 4; ++i) ptx::mbar_init(bar(i), 1);
    ptx::mbar_init(phi_ready, 128);
    ptx::mbar_init(phi_free, 1);
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
  const uint32_t tmem_base = *tmem_holder;
  auto wait_uniform = [&](uint32_t bar_addr, uint32_t parity) {
    const int ok = ptx::mbar_wait(bar_addr, parity, abort_flag) ? 1 : 0;
    return __all_sync(0xffffffffu, ok) != 0;
  };
  auto wait_tmem = [&](uint32_t bar_addr, uint32_t parity) {
    const bool up = wait_uniform(bar_addr, parity);
    if (up) ptx::tc_fence_after();
    return up;
  };
  auto load_row = [&](const RawRows& t, int tok, float (&v)[D]) {
    uint4 w[D / 8];
#pragma unroll
    for (int j = 0; j < D / 8; ++j) w[j] = make_uint4(0u, 0u, 0u, 0u);
    if (tok < p.n_tokens) {
      const uint4* src = reinterpret_cast<const uint4*>(t.ptr + b * t.sb + h * t.sh + tok * t.sn);
#pragma unroll
      for (int j = 0; j < D / 8; ++j) w[j] = __ldg(src + j);
    }
#pragma unroll
    for (int j = 0; j < D / 8; ++j) {
      const uint32_t u[4] = {w[j].x, w[j].y, w[j].z, w[j].w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        v[8 * j + 2 * c] = ptx::bf16_lo(u[c]);
        v[8 * j + 2 * c + 1] = ptx::bf16_hi(u[c]);
      }
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
    const uint32_t x_k = ptx::desc_lo(x_addr, 16), y_k = ptx::desc_lo(y_addr, 16), y_mn = ptx::desc_lo(y_addr, kGroupBytes);
    const uint32_t zb_k = ptx::desc_lo(zb_addr, 16), zb_mn = ptx::desc_lo(zb_addr, cfg::ZB_GROUP);
    auto k_step = [](int kk, int group) { return static_cast<uint32_t>(((kk >> 2) * group + (kk & 3) * 32) >> 4); };
    auto half_step = [](int kk) { return static_cast<uint32_t>((kk >> 2) * 64 + (kk & 3) * 8); };  // 16-bit tile, in two halves
    for (int i = 0; i < n_iter; ++i) {
      const bool last = i + 1 == n_iter, have_z = i > 0;
      const uint32_t b_k = ptx::desc_lo(b_tile(i), 16), b_mn = ptx::desc_lo(b_tile(i), kGroupBytes);
      const uint32_t a_k = ptx::desc_lo(a_tile(i), 16);
      if (!wait_uniform(phi_ready, i & 1)) break;
      if (!wait_uniform(full_bar(i), (i >> 1) & 1)) break;
      if (want_dx && have_z && !wait_uniform(dx_free, (i - 1) & 1)) break;  // the score tile's place is free
      ptx::tc_fence_after();
      if (leader) {
        ptx::mma_ss(tP, x_k, y_k, ptx::kDescHi, IDESC_P, 0u);
        if (want_dx) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            ptx::mma_ss(tT, a_k + k_step(kk, 0), b_k + k_step(kk, 0), ptx::kDescHi, IDESC_P, kk > 0 ? 1u : 0u);
        }
        ptx::tc_commit(p_full);
      }
      if (have_z) {
        if (!wait_uniform(zb_ready, (i - 1) & 1)) break;
        if (want_o && !wait_uniform(o_free, (i - 1) & 1)) break;
        ptx::tc_fence_after();
      }
      if (leader) {
        if (want_o && have_z) {
#pragma unroll
          for (int kk = 0; kk < NF / 16; ++kk)
            ptx::mma_ss(tO, x_k + k_step(kk, kGroupBytes), zb_k + k_step(kk, cfg::ZB_GROUP), ptx::kDescHi, IDESC_XZ, kk > 0 ? 1u : 0u);
        }
        if (!last) {
          // The instruction spans 128 rows of Z; the upper 64 read what follows the b tile in shared memory
          // and land in tensor-memory lanes nobody reads.
#pragma unroll
          for (int kk = 0; kk < kChunk / 16; ++kk)
            ptx::mma_ss(tZ, b_mn + kk * (2048 >> 4), y_mn + kk * (2048 >> 4), ptx::kDescHi, IDESC_Z, (have_z || kk > 0) ? 1u : 0u);
          if (!want_dx) ptx::tc_commit(z_full);
        }
      }
      if (!wait_tmem(pb_ready, i & 1)) break;
      if (leader) {
        if (want_o) {
#pragma unroll
          for (int kk = 0; kk < kChunk / 16; ++kk)
            ptx::mma_ts(tO, tP + half_step(kk), b_mn + kk * (2048 >> 4), ptx::kDescHi, IDESC_PB, (have_z || kk > 0) ? 1u : 0u);
          ptx::tc_commit(o_full);
        }
        if (want_dx) {
          if (have_z) {  // into the place of the scores, which the conversion and f(s) b have used up
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              ptx::mma_ss(tP, a_k + k_step(kk, 0), zb_mn + kk * (2048 >> 4), ptx::kDescHi, IDESC_AZ, kk > 0 ? 1u : 0u);
          }
#pragma unroll
          for (int kk = 0; kk < kChunk / 16; ++kk)
            ptx::mma_ts(tTy, tT + half_step(kk), y_mn + kk * (2048 >> 4), ptx::kDescHi, IDESC_TY, kk > 0 ? 1u : 0u);
          ptx::tc_commit(dx_full);
          if (!last) ptx::tc_commit(z_full);
        }
        ptx::tc_commit(phi_free);
        ptx::tc_commit(empty_bar(i));
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
#pragma unroll
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
        // kept columns of this row, a bit each
        uint32_t keep = 0xffffffffu;
        if (cb == quad) keep = upper_flag ? 0xffffffffu << lane : 0xffffffffu >> (31 - lane);
        if (want_o) {
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            float f[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const float s = cs * __uint_as_float(rs[2 * c + u]);
              f[u] = (keep >> (2 * c + u)) & 1u ? 1.f + s * (1.f + 0.5f * s) : 0.f;
            }
            pk[c] = ptx::pack_bf16x2(f[0], f[1]);
          }
          ptx::tmem_st16(dst_s, pk);
        }
        if (want_dx) {
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            float t[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const float s = cs * __uint_as_float(rs[2 * c + u]);
              t[u] = (keep >> (2 * c + u)) & 1u ? __uint_as_float(rt[2 * c + u]) * (cs + cs * s) : 0.f;
            }
            pk[c] = ptx::pack_bf16x2(t[0], t[1]);
          }
          ptx::tmem_st16(dst_t, pk);
        }
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
        float xv[D], acc[D];
        load_row(pr.x, tok, xv);
        if (!wait_tmem(dx_full, i & 1)) break;
        ptx::tmem_ld32(lane_base + cfg::TY_COL, ra);  // (16 columns of it)
#pragma unroll
        for (int a = 0; a < D; ++a) acc[a] = __uint_as_float(ra[a]);
        if (i > 0) {
          ptx::static_for<NF / 32>([&](auto cb_c) {
            constexpr int CB = decltype(cb_c)::value;
            ptx::tmem_ld32(lane_base + cfg::P_COL + CB * 32, ra);
            ptx::static_for<32>([&](auto c) {
              constexpr int C = decltype(c)::value, F = CB * 32 + C;
              const float gv = __uint_as_float(ra[C]);
              if constexpr (F < D) {
                acc[F] += gv;
              } else if constexpr (F >= 16 && F < 16 + cfg::PAIRS) {
                constexpr int A = cfg::first(F - 16), B = cfg::second(F - 16);
                acc[A] += gv * xv[B];
                acc[B] += gv * xv[A];
              }
            });
          });
        }
        if (tok < p.n_tokens) {
          uint4* dst = reinterpret_cast<uint4*>(const_cast<__nv_bfloat16*>(pr.dx.ptr) + b * pr.dx.sb + h * pr.dx.sh + tok * pr.dx.sn);
#pragma unroll
          for (int j = 0; j < D / 8; ++j)
            dst[j] = make_uint4(ptx::pack_bf16x2(acc[8 * j], acc[8 * j + 1]), ptx::pack_bf16x2(acc[8 * j + 2], acc[8 * j + 3]),
                                ptx::pack_bf16x2(acc[8 * j + 4], acc[8 * j + 5]), ptx::pack_bf16x2(acc[8 * j + 6], acc[8 * j + 7]));
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
    float xv[D], yv[D];
    load_row(pr.y, mem_chunk(0) * kChunk + r, yv);
    load_row(pr.x, mem_chunk(0) * kChunk + r, xv);
    auto write_row = [&](uint32_t tile, const float (&v)[D], auto pieces) {
      ptx::static_for<decltype(pieces)::value>([&](auto piece) {
        constexpr int P = decltype(piece)::value;
        uint32_t w[4];
        ptx::static_for<4>([&](auto c) {
          constexpr int F = 8 * P + 2 * decltype(c)::value;
          auto feature = [&](auto f_c) -> float {
            constexpr int FC = decltype(f_c)::value;
            if constexpr (FC < D) {
              return v[FC];
            } else if constexpr (FC >= 16 && FC < 16 + cfg::PAIRS) {
              constexpr int A = cfg::first(FC - 16), B = cfg::second(FC - 16);
              return v[A] * v[B];
            } else {
              return FC == 16 + cfg::PAIRS ? 1.f : 0.f;
            }
          };
          w[(F >> 1) & 3] = ptx::pack_bf16x2(feature(std::integral_constant<int, F>{}), feature(std::integral_constant<int, F + 1>{}));
        });
        ptx::st_shared_v4(tile + (P >> 3) * kGroupBytes + r * 128 + (((P & 7) ^ swz) << 4), w[0], w[1], w[2], w[3]);
      });
    };
    for (int i = 0; i < n_iter; ++i) {
      if (i > 0 && !wait_uniform(phi_free, (i - 1) & 1)) break;
      write_row(y_addr, yv, std::integral_constant<int, NF / 8>{});
      if (want_o) write_row(x_addr, xv, std::integral_constant<int, NF / 8>{});
      else write_row(x_addr, xv, std::integral_constant<int, 2>{});  // scores need the raw columns only
      ptx::fence_proxy_async_smem();
      ptx::mbar_arrive(phi_ready);
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
