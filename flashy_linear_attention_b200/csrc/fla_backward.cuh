// All three gradients of causal linear attention (dk = dv <= 128) in one sweep of one CTA per head, for
// sm_100a. Replaces flashlinear/kernels/linear_attn_kernels.py:103-307 where there are heads enough.
//
// fla_kernel.cuh computes the gradients as three products, each in a CTA of its own: together they load
// nine tiles a chunk, write three and run twelve MMA groups. Here one CTA walks the chunks from the last to the
// first, loads q, k, v and dO (g) once each, and carries both states in tensor memory (fp32, dk x dv):
//     R = sum of q^T g over the chunks after this one           (grows)
//     S = sum of k^T v over the chunks before this one          (starts as the forward's final state)
// Per 128-token chunk, in issue order (eleven groups of eight 128 x D x 16 MMAs at D = 128):
//     P = v g^T (j <= i kept),  S -= k^T v,   dK = v R^T + P q
//     P = k q^T (same mask),    R += q^T g,   dV = k R   + P g
//     P = g v^T,                              dQ = g S^T + P k
// S is exclusive of the chunk when dQ uses it: no difference of two sums over the chunk is left in dQ. The
// groups between a score tile and the product that consumes it cover its conversion, and those before the
// accumulator is written again cover its drain; at D = 64 there are two of each in tensor memory, at
// D = 128 S, R, P and the accumulator fill its 512 columns. The states' 16-bit copies serve as MMA operands in
// either direction (dV contracts over R's rows, dK over its columns) without a second copy.
//
// At D = 128 a chunk moves 1.0 MB of operands, states, tiles and staged outputs through an SM's shared memory, at
// least 8000 cycles at 128 bytes, against 6300 of MMAs (three CTAs of fla_chunk_kernel: 1.25 MB). It takes
// 10600 to 11200 (346 - 365 us for 64 chunks): the rest are waits for tiles and score conversions that nothing
// covers with one score tile and one accumulator. At D = 64 5700 cycles, the issuer's waits and the
// conversions. (Counters: tensor pipe 64 % and 53 % of active cycles, DRAM 62 % and 55 % of its peak.)
// 128 heads, in one CTA each / three: 4096 x 128 186 / 220 us, 8192 x 128 365 / 422 us, 4096 x 64 93 / 125 us.
// NORM 4096 x 128: 308 us, its loads of d and the chunk vectors lie behind the waits for the tiles they go with
// (tensor pipe 33 %, DRAM 36 %). dQ's error against 64 bits 2.34e-3 / 2.40e-3.
//
// CTA layout (608 threads, one CTA per SM):
//   warps 0, 18   TMA producers, each half of every tile (see fla_kernel.cuh)
//   warp 1        MMA issuer (one elected lane) and TMEM owner
//   warps 2-9     converters of the scores: fp32 -> mask -> 16 bits, in place (TMEM); before the loop, the
//                 states at the start
//   warps 10-13   epilogue: accumulator -> 16 bits -> staging -> TMA store
//   warps 14-17   converters of the states: fp32 (TMEM) -> 16 bits (shared memory). With one group for scores
//                 and states its five conversions a chunk, one behind the other, were the chunk period.
#pragma once
#include "fla_kernel.cuh"

namespace fla {

struct BackwardParams {
  CUtensorMap q, k, v, g;     // 4-D maps, boxes as in Problem
  CUtensorMap dq, dk, dv;     // boxes of 64 columns x 32 rows
  // states, fp32 [bh][dk][dk]: S after this call's tokens; R before them (null: zero); R including them (or null)
  const float* s_last;
  const float* r_init;
  float* r_final;
  int dim;                    // dk
  int first_exact;            // nothing precedes token 0: the first chunk's S is zero, and is not used
  int heads, nchunks, n_tokens;
  int* status;                // see KernelParams
  unsigned wait_limit_us;
  int debug_withhold;
  // ---- NORM: the gradient of the attention's denominator in the same pass. With g the gradient of the product
  // (dnum) and d_i that of the denominator of token i,
  //     dQ_i += d_i sum_{j<=i} k_j,    dK_j += sum_{i>=j} d_i q_i.
  // Inside the chunk d_i is a bias on the scores g_i . v_j of both, in fp32, before they are rounded; what
  // comes from the other chunks is a vector per chunk, added in fp32 before the result is rounded.
  const float* d;             // [bh][tokens]
  const float* zk;            // [bh][chunks][dk]: sum of k over the chunks before
  const float* zq;            // [bh][chunks][dk]: sum of d_i q_i over the chunks after
};

constexpr int kBwdThreads = 608;

template <int D>
struct BwdCfg {
  static_assert(D == 64 || D == 128, "unsupported head dim");
  static constexpr int G = D / 64;                      // 64-column groups of a tile
  static constexpr int TILE_BYTES = G * kGroupBytes;
  static constexpr int LOAD_ROWS = Cfg<D, D>::LOAD_ROWS;
  static constexpr int STATE_BYTES = G * D * 128;       // 16-bit copy of a state
  // D = 128: four slots, one for each tile of a chunk. They are released in the order q, v, g, k and taken by the
  // next chunk's tiles in the order of their first use, v, g, k, q, so a tile has a third of a chunk's time
  // or more to arrive. (A fifth slot, with the outputs staged in the states' copies while those are dead,
  // was slower: the copy of S then waits for dK to leave it, 1000 cycles a chunk.)
  static constexpr int NSLOT = D == 128 ? 4 : 8;
  static constexpr int STAGE_BYTES = D == 128 ? TILE_BYTES : 3 * kGroupBytes;  // D = 64: one stage per gradient
  static constexpr int BAR_BYTES = 512;
  static constexpr int SB_OFF = NSLOT * TILE_BYTES;
  static constexpr int RB_OFF = SB_OFF + STATE_BYTES;
  static constexpr int STAGE_OFF = RB_OFF + STATE_BYTES;
  // 32 KB for the transposes of the states at the start (and, four warps, of R at the end): the stage
  static constexpr int SCRATCH_OFF = STAGE_OFF;
  static_assert(STAGE_BYTES >= 8 * 4096, "scratch of load_state()");
  static constexpr int BAR_OFF = STAGE_OFF + STAGE_BYTES;
  static constexpr int SMEM_BYTES = 1024 + BAR_OFF + BAR_BYTES;
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
  static constexpr int NBARS = 2 * NSLOT + 15;
  static_assert(NBARS * 8 + 16 <= BAR_BYTES, "barrier area");
  // tensor memory columns: fp32 scores, 128 each (their 16-bit form replaces each half in place), output
  // accumulators and states. D = 64 leaves room for two score tiles and two accumulators.
  static constexpr bool DOUBLE = D == 64;
  __device__ static constexpr int p_col(int n) { return DOUBLE ? (n & 1) * 128 : 0; }
  __device__ static constexpr int o_col(int n) { return DOUBLE ? 256 + (n & 1) * 64 : 128; }
  static constexpr int S_COL = DOUBLE ? 384 : 256, R_COL = S_COL + D;
  static constexpr int TMEM_COLS = 512;
};

// R -> the caller's array, a state-converter warp's 32 rows, at D = 128 through a 32 x 32 transpose in
// `scratch` (4 KB a warp) so that global stores are whole 128-byte row segments. Out of line: once a CTA.
template <int D>
__device__ __noinline__ void write_final_rows(float* dst, int dim, uint32_t state, uint32_t scratch, int quad) {
  const int lane = static_cast<int>(threadIdx.x & 31), row = quad * 32 + lane;
  uint32_t r[32];
#pragma unroll 1
  for (int cb = 0; cb < D / 32; ++cb) {
    ptx::tmem_ld32(state + cb * 32, r);
    if (D == 128) {
#pragma unroll
      for (int j = 0; j < 32; ++j) ptx::st_shared_b32(scratch + (j * 32 + (lane ^ j)) * 4, r[j]);
      __syncwarp();
      const int col = cb * 32 + lane;
#pragma unroll 4
      for (int rr = 0; rr < 32; ++rr) {
        const int grow = quad * 32 + rr;
        const uint32_t x = ptx::ld_shared_b32(scratch + (lane * 32 + (rr ^ lane)) * 4);
        if (grow < dim && col < dim) dst[static_cast<size_t>(grow) * dim + col] = __uint_as_float(x);
      }
      __syncwarp();
    } else if (row < dim) {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (cb * 32 + j < dim) dst[static_cast<size_t>(row) * dim + cb * 32 + j] = __uint_as_float(r[j]);
    }
  }
}

// One group of MMAs, 4 * blocks steps of 16 along the contraction: from step to step the operands' addresses
// (descriptor words, or the tensor-memory address of a) advance by `step`, from block to block by `jump`.
struct Walk {
  uint32_t start, step, jump;
};
template <bool TS>
__device__ __forceinline__ void issue_group(bool leader, uint32_t d, Walk a, Walk b, uint32_t idesc, uint32_t accumulate, int blocks) {
#pragma unroll
  for (int blk = 0; blk < blocks; ++blk) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t av = a.start + blk * a.jump + j * a.step, bv = b.start + blk * b.jump + j * b.step;
      const uint32_t add = (blk > 0 || j > 0) ? 1u : accumulate;
      if (TS) ptx::mma_ts_on(leader, d, av, bv, ptx::kDescHi, idesc, add);
      else ptx::mma_ss_on(leader, d, av, bv, ptx::kDescHi, idesc, add);
    }
  }
}

// A state at the start -> tensor memory (fp32, `state`: this warp's lane quadrant) and, with `copy`, the 16-bit
// operand copy. A warp moves its 32 rows and half of the columns, in 32 x 32 blocks through `scratch` (4 KB a
// warp), so that global loads are whole 128-byte row segments; what lies beyond dim x dim is zero. Out of
// line: once or twice a CTA.
template <int D, bool HALF>
__device__ __noinline__ void load_state(const float* src, int dim, uint32_t state, uint32_t copy, uint32_t scratch, int quad, int half) {
  const int lane = static_cast<int>(threadIdx.x & 31), row = quad * 32 + lane;
  uint32_t r[32];
#pragma unroll 1
  for (int jb = 0; jb < D / 64; ++jb) {
    const int cb = half * (D / 64) + jb, col = cb * 32 + lane;
#pragma unroll
    for (int rr = 0; rr < 32; ++rr) {
      const int grow = quad * 32 + rr;
      const bool valid = grow < dim && col < dim;
      r[rr] = ptx::ld_global_cg_b32(src + (valid ? static_cast<size_t>(grow) * dim + col : 0));
      r[rr] = valid ? r[rr] : 0u;
    }
#pragma unroll
    for (int rr = 0; rr < 32; ++rr) ptx::st_shared_b32(scratch + (lane * 32 + (rr ^ lane)) * 4, r[rr]);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 32; ++j) r[j] = ptx::ld_shared_b32(scratch + (j * 32 + (lane ^ j)) * 4);
    __syncwarp();
    ptx::tmem_st32(state + cb * 32, r);
    if (copy != 0 && row < D) {
#pragma unroll
      for (int jj = 0; jj < 4; ++jj)
        ptx::st_shared_v4(copy + (cb >> 1) * (D * 128) + row * 128 + ((((cb & 1) * 4 + jj) ^ (row & 7)) << 4),
                          ptx::pack16x2<HALF>(__uint_as_float(r[jj * 8 + 0]), __uint_as_float(r[jj * 8 + 1])),
                          ptx::pack16x2<HALF>(__uint_as_float(r[jj * 8 + 2]), __uint_as_float(r[jj * 8 + 3])),
                          ptx::pack16x2<HALF>(__uint_as_float(r[jj * 8 + 4]), __uint_as_float(r[jj * 8 + 5])),
                          ptx::pack16x2<HALF>(__uint_as_float(r[jj * 8 + 6]), __uint_as_float(r[jj * 8 + 7])));
    }
  }
  ptx::tc_wait_st();
  ptx::fence_proxy_async_smem();
  ptx::tc_fence_before();
}

template <int D, bool HALF, bool NORM = false>
__global__ void __launch_bounds__(kBwdThreads, 1)
fla_backward_kernel(const __grid_constant__ BackwardParams p) {
  using cfg = BwdCfg<D>;
  constexpr int NSLOT = cfg::NSLOT;
  extern __shared__ uint8_t smem_raw[];

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // provably warp-uniform
  const int lane = threadIdx.x & 31;
  const int bh = blockIdx.z;
  const int h = bh % p.heads, b = bh / p.heads;

  const uint32_t raw_addr = ptx::smem_u32(smem_raw);
  const uint32_t smem_base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - raw_addr);
  const uint32_t sb_addr = smem_base + cfg::SB_OFF, rb_addr = smem_base + cfg::RB_OFF;
  const uint32_t bar_base = smem_base + cfg::BAR_OFF;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (NSLOT + s); };
  auto bar = [&](int i) { return bar_base + 8u * (2 * NSLOT + i); };
  // The three products of a chunk, dK, dV and dQ, are numbered through: n = 3 i + 0, 1, 2. What is signalled
  // once a product alternates between two barriers, so that a wait is never overtaken (see fla_kernel.cuh).
  auto p_full = [&](int n) { return bar(n & 1); };          // score tile complete
  auto pb_ready = [&](int n) { return bar(2 + (n & 1)); };  // its 16-bit form written (256 arrivals)
  auto o_full = [&](int n) { return bar(4 + (n & 1)); };    // output complete
  auto o_free = [&](int n) { return bar(6 + (n & 1)); };    // and read (128)
  const uint32_t s_full = bar(8);     // S of this chunk is complete
  const uint32_t sb_ready = bar(9);   // and its 16-bit copy written (128)
  const uint32_t r_full = bar(10);    // R including this chunk is complete
  const uint32_t rb_ready = bar(11);  // and its 16-bit copy written (128)
  const uint32_t s_loaded = bar(12), r_loaded = bar(13);  // S, R at the start are in tensor memory (256)
  const uint32_t drained = bar(14);   // everything the issuer issued has completed
  volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(smem_gen + cfg::BAR_OFF + cfg::NBARS * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + cfg::BAR_OFF + cfg::NBARS * 8 + 4);

  const int n_iter = p.nchunks;
  auto mem_chunk = [&](int i) { return n_iter - 1 - i; };
  const bool has_r = p.r_init != nullptr;  // R does not start from zero

  // ------------------------------------------------------------------ setup
  if (threadIdx.x == 0) {
    abort_flag[0] = 0;
    abort_flag[1] = static_cast<int>(p.wait_limit_us);
    for (int s = 0; s < NSLOT; ++s) {
      ptx::mbar_init(full_bar(s), 2);  // both producers
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int n = 0; n < 2; ++n) {
      ptx::mbar_init(p_full(n), 1);
      ptx::mbar_init(pb_ready(n), 256);
      ptx::mbar_init(o_full(n), 1);
      ptx::mbar_init(o_free(n), 128);
    }
    ptx::mbar_init(s_full, 1);
    ptx::mbar_init(sb_ready, 128);
    ptx::mbar_init(r_full, 1);
    ptx::mbar_init(rb_ready, 128);
    ptx::mbar_init(s_loaded, 256);
    ptx::mbar_init(r_loaded, 256);
    ptx::mbar_init(drained, 1);
    ptx::fence_barrier_init();
    ptx::fence_proxy_async_smem();
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_holder)), cfg::TMEM_COLS);
    ptx::tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    ptx::prefetch_tensormap(&p.q);
    ptx::prefetch_tensormap(&p.k);
    ptx::prefetch_tensormap(&p.v);
    ptx::prefetch_tensormap(&p.g);
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_holder, 0);

  auto wait_uniform = [&](uint32_t bar_addr, uint32_t parity) {
    const int ok = ptx::mbar_wait(bar_addr, parity, abort_flag) ? 1 : 0;
    return __all_sync(0xffffffffu, ok) != 0;
  };
  auto wait_tmem = [&](uint32_t bar_addr, uint32_t parity) {
    const bool up = wait_uniform(bar_addr, parity);
    if (up) ptx::tc_fence_after();
    return up;
  };
  // Chunk i has tiles v, g, k, q (w = 0 .. 3), in the order of their first use: at D = 64 along the ring, at
  // D = 128 in the slots in turn. use(): how often the slot was filled before.
  constexpr int V = 0, G = 1, K = 2, Q = 3;
  auto slot_of = [&](int i, int w) { return cfg::DOUBLE ? (4 * i + w) % NSLOT : (w - i) & 3; };
  auto use_of = [&](int i, int w) { return cfg::DOUBLE ? (4 * i + w) / NSLOT : i; };
  auto slot_addr = [&](int s) { return smem_base + static_cast<uint32_t>(s) * cfg::TILE_BYTES; };

  if (warp == 0 || warp == 18) {
    // ================================================================ TMA producers
    const bool leader = ptx::elect_one();
    const int part = warp == 0 ? 0 : 1;
    constexpr int kPartBytes = cfg::TILE_BYTES / 2;
    const int part_col = cfg::G == 2 ? part * 64 : 0;
    const int part_row = cfg::G == 2 ? 0 : part * cfg::LOAD_ROWS;
    for (int t = 0; t < 4 * n_iter; ++t) {
      const int i = t >> 2, w = t & 3;
      const int s = slot_of(i, w);
      if (!wait_uniform(empty_bar(s), (use_of(i, w) & 1) ^ 1u)) break;
      const int tok = mem_chunk(i) * kChunk + part_row;
      const CUtensorMap* map = w == V ? &p.v : w == G ? &p.g : w == K ? &p.k : &p.q;
      if (leader) {
        ptx::mbar_expect_tx(full_bar(s), kPartBytes);
        if (!(p.debug_withhold && t == 0))
          ptx::tma_load_4d(slot_addr(s) + part * kPartBytes, map, full_bar(s), part_col, tok, h, b);
        // At D = 128 a slot is free only shortly before its tile is wanted: the tile after that comes into L2
        // now. (128 heads x 8192, an earlier state of the kernel: 396 us without, 376 with; at D = 64, two chunks
        // deep, no difference.)
        if (D == 128 && i + 1 < n_iter) ptx::tma_prefetch_4d(map, part_col, tok - kChunk, h, b);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    // ================================================================ MMA issuer
    constexpr uint32_t IDESC_P = ptx::make_idesc(128, kChunk, false, false, HALF);  // a b^T over the head dim
    constexpr uint32_t IDESC_ADD = ptx::make_idesc(128, D, true, true, HALF);       // state += a^T b
    constexpr uint32_t IDESC_SUB = IDESC_ADD | (1u << 13);                          // (A negated)
    constexpr uint32_t IDESC_XT = ptx::make_idesc(128, D, false, false, HALF);      // a X^T: contracts X's columns
    constexpr uint32_t IDESC_X = ptx::make_idesc(128, D, false, true, HALF);        // a X, P b: contracts rows
    const uint32_t tS = tmem_base + cfg::S_COL, tR = tmem_base + cfg::R_COL;
    const bool leader = ptx::elect_one();
    auto wait = [&](uint32_t bar_addr, uint32_t parity) { return wait_uniform(bar_addr, parity); };
    auto commit = [&](uint32_t bar_addr) { ptx::tc_commit_on(leader, bar_addr); };
    // Operands: a chunk tile or a state's copy, contracted over its columns (K-major) or its rows (MN-major).
    constexpr int kStateGroup = D * 128;  // bytes between the 64-column groups of a state's copy
    auto columns = [](uint32_t addr, int group) { return Walk{ptx::desc_lo(addr, 16), 32u >> 4, static_cast<uint32_t>(group) >> 4}; };
    auto rows = [](uint32_t addr, int group) { return Walk{ptx::desc_lo(addr, group), 2048u >> 4, 8192u >> 4}; };
    auto scores = [&](int n, uint32_t a, uint32_t bt) {  // P = a b^T
      issue_group<false>(leader, tmem_base + cfg::p_col(n), columns(a, kGroupBytes), columns(bt, kGroupBytes), IDESC_P, 0u, D / 64);
      commit(p_full(n));
    };
    // For D = 64 the instruction still spans 128 rows of the state; the upper 64 read whatever follows the a
    // tile in shared memory and land in tensor-memory lanes nobody reads.
    auto state_add = [&](uint32_t t_state, uint32_t a, uint32_t bt, uint32_t idesc, bool accumulate) {
      issue_group<false>(leader, t_state, rows(a, kGroupBytes), rows(bt, kGroupBytes), idesc, accumulate ? 1u : 0u, 2);
    };
    auto times_state_t = [&](int n, uint32_t a, uint32_t x) {  // O = a X^T
      issue_group<false>(leader, tmem_base + cfg::o_col(n), columns(a, kGroupBytes), columns(x, kStateGroup), IDESC_XT, 0u, D / 64);
    };
    auto times_state = [&](int n, uint32_t a, uint32_t x) {  // O = a X
      issue_group<false>(leader, tmem_base + cfg::o_col(n), columns(a, kGroupBytes), rows(x, kStateGroup), IDESC_X, 0u, D / 64);
    };
    auto times_scores = [&](int n, uint32_t bt, bool accumulate) {  // O += P b, P in its 16-bit form (two halves)
      issue_group<true>(leader, tmem_base + cfg::o_col(n), Walk{tmem_base + cfg::p_col(n), 8u, 64u}, rows(bt, kGroupBytes), IDESC_X, accumulate ? 1u : 0u, 2);
      commit(o_full(n));
    };

    bool ok = wait(s_loaded, 0);
    auto tile = [&](int i, int w) { return slot_addr(slot_of(i, w)); };
    auto wait_tile = [&](int i, int w) { return wait(full_bar(slot_of(i, w)), use_of(i, w) & 1); };
    auto release = [&](int i, int w) { commit(empty_bar(slot_of(i, w))); };
    auto scores_k = [&](int i) {
      if (!wait_tile(i, V) || !wait_tile(i, G)) return false;
      ptx::tc_fence_after();
      scores(3 * i, tile(i, V), tile(i, G));
      return true;
    };
    auto scores_v = [&](int i) {
      if (!wait_tile(i, K) || !wait_tile(i, Q)) return false;
      ptx::tc_fence_after();
      scores(3 * i + 1, tile(i, K), tile(i, Q));
      return true;
    };
    auto scores_q = [&](int i) {
      scores(3 * i + 2, tile(i, G), tile(i, V));
      release(i, V);
    };
    auto wait_scores = [&](int n) {
      const bool up = wait(pb_ready(n), (n >> 1) & 1);
      ptx::tc_fence_after();
      return up;
    };
    auto wait_output = [&](int n) {  // the accumulator of product n has been drained of the one before
      const int before = n - (cfg::DOUBLE ? 2 : 1);
      if (before < 0) return true;
      const bool up = wait(o_free(before), (before >> 1) & 1);
      ptx::tc_fence_after();
      return up;
    };
    // Where two score tiles fit, the scores of a product are issued before its predecessor's are waited for.
    if (cfg::DOUBLE) ok = ok && scores_k(0);
    for (int i = 0; ok && i < n_iter; ++i) {
      const int n = 3 * i;
      const bool have_r = i > 0 || has_r;
      const bool use_s = !(p.first_exact && mem_chunk(i) == 0);
      const bool want_r = i + 1 < n_iter || p.r_final != nullptr;
      // ---- dK
      if (!(cfg::DOUBLE ? scores_v(i) : scores_k(i))) break;
      // S -= k^T v. The converters read the previous S before sb_ready, which was waited for.
      if (!cfg::DOUBLE && !wait_tile(i, K)) break;
      state_add(tS, tile(i, K), tile(i, V), IDESC_SUB, true);
      commit(s_full);
      if (have_r && !(i > 0 ? wait(rb_ready, (i - 1) & 1) : wait(r_loaded, 0))) break;
      if (!wait_output(n)) break;
      ptx::tc_fence_after();
      if (have_r) times_state_t(n, tile(i, V), rb_addr);
      if (!wait_scores(n)) break;
      if (!cfg::DOUBLE && !wait_tile(i, Q)) break;
      times_scores(n, tile(i, Q), have_r);
      // ---- dV
      if (cfg::DOUBLE) scores_q(i);
      else scores(n + 1, tile(i, K), tile(i, Q));
      // R += q^T g. The converters read the previous R before rb_ready.
      if (want_r) {
        state_add(tR, tile(i, Q), tile(i, G), IDESC_ADD, have_r);
        commit(r_full);
      }
      release(i, Q);
      if (!wait_output(n + 1)) break;
      if (have_r) times_state(n + 1, tile(i, K), rb_addr);
      if (!wait_scores(n + 1)) break;
      times_scores(n + 1, tile(i, G), have_r);
      // ---- dQ
      if (!cfg::DOUBLE) scores_q(i);
      else if (i + 1 < n_iter && !scores_k(i + 1)) break;
      if (!wait(sb_ready, i & 1)) break;
      if (!wait_output(n + 2)) break;
      ptx::tc_fence_after();
      if (use_s) times_state_t(n + 2, tile(i, G), sb_addr);
      release(i, G);
      if (!wait_scores(n + 2)) break;
      times_scores(n + 2, tile(i, K), use_s);
      release(i, K);
    }
    // Nobody waits for the last releases; the barriers have to outlive them all the same.
    commit(drained);
  } else if (warp < 10) {
    // ================================================================ converters of the scores
    const int half = (warp - 2) >> 2;  // column half this group owns
    const int quad = warp & 3;         // TMEM lane quadrant this warp may access
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    {
      // (transposes go through the stage: nothing is staged before both states are in place)
      const size_t offset = static_cast<size_t>(bh) * p.dim * p.dim;
      const uint32_t scratch = smem_base + cfg::SCRATCH_OFF + static_cast<uint32_t>(warp - 2) * 4096u;
      load_state<D, HALF>(p.s_last + offset, p.dim, lane_base + cfg::S_COL, 0u, scratch, quad, half);
      ptx::mbar_arrive(s_loaded);
      if (has_r) {
        load_state<D, HALF>(p.r_init + offset, p.dim, lane_base + cfg::R_COL, rb_addr, scratch, quad, half);
        ptx::mbar_arrive(r_loaded);
      }
    }
    uint32_t ra[32], rb[32];
    for (int n = 0; n < 3 * n_iter; ++n) {
      // fp32 -> mask -> 16 bits, this group's 64 columns into the first half of their own place. Relative
      // to the warp's 32 rows a block of 32 columns is kept, masked, or (block index == quadrant) the
      // diagonal one. dK, dV: columns from the row on are kept (all but those up to the row before); dQ:
      // columns up to the row.
      const bool upper = n % 3 != 2;
      const int cb0 = half * 2, cb1 = half * 2 + 1;
      const bool masked0 = upper ? (cb0 < quad) : (cb0 > quad);  // warp-uniform
      const bool masked1 = upper ? (cb1 < quad) : (cb1 > quad);
      const int edge = upper ? lane - 1 : lane;
      const uint32_t flip = upper ? 0xffffffffu : 0u;
      const uint32_t src = lane_base + cfg::p_col(n) + half * 64;
      const int tok0 = mem_chunk(n / 3) * kChunk;
      const float* d = NORM ? p.d + static_cast<size_t>(bh) * p.n_tokens : nullptr;
      float d_row = 0.f;
      if (NORM && n % 3 == 2) {  // scores of dQ: a bias per row
        const int tok = tok0 + quad * 32 + lane;
        if (tok < p.n_tokens) d_row = __ldg(d + tok);
      }
      if (!wait_tmem(p_full(n), (n >> 1) & 1)) break;
      if (!masked0 && !masked1) ptx::tmem_ld32x2(src, ra, src + 32, rb);
      else if (!masked0) ptx::tmem_ld32(src, ra);
      else if (!masked1) ptx::tmem_ld32(src + 32, rb);
      auto convert_block = [&](int cb, bool masked, uint32_t (&r)[32]) {
        uint32_t pk[16];
        if (masked) {
#pragma unroll
          for (int j = 0; j < 16; ++j) pk[j] = 0u;
        } else {
          if (NORM && n % 3 == 0) {  // of dK: a bias per column (the token count is a multiple of 4)
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const int tok = tok0 + cb * 32 + j;
              float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
              if (tok < p.n_tokens) x = __ldg(reinterpret_cast<const float4*>(d + tok));
              r[j] = __float_as_uint(__uint_as_float(r[j]) + x.x);
              r[j + 1] = __float_as_uint(__uint_as_float(r[j + 1]) + x.y);
              r[j + 2] = __float_as_uint(__uint_as_float(r[j + 2]) + x.z);
              r[j + 3] = __float_as_uint(__uint_as_float(r[j + 3]) + x.w);
            }
          } else if (NORM) {
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + d_row);
          }
#pragma unroll
          for (int j = 0; j < 16; ++j)
            pk[j] = ptx::pack16x2<HALF>(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
          if (cb == quad) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
              pk[j] &= (edge > 2 * j ? 0xffffffffu : edge == 2 * j ? 0x0000ffffu : 0u) ^ flip;
          }
        }
        ptx::tmem_st16(src + (cb & 1) * 16, pk);
      };
      convert_block(cb0, masked0, ra);
      convert_block(cb1, masked1, rb);
      ptx::tc_wait_st();
      ptx::tc_fence_before();
      ptx::mbar_arrive(pb_ready(n));
    }
  } else if (warp < 14) {
    // ================================================================ epilogue
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t swz = static_cast<uint32_t>(row & 7);
    const uint32_t own_stage = smem_base + cfg::STAGE_OFF;
    uint32_t ra[32], rb[32];
    for (int n = 0; n < 3 * n_iter; ++n) {
      // One output: 128 rows of this chunk through a stage to global memory. Every warp moves its own 32 rows.
      const int which = n % 3;  // 0: dK, 1: dV, 2: dQ
      const CUtensorMap* map = which == 0 ? &p.dk : which == 1 ? &p.dv : &p.dq;
      const uint32_t stage = own_stage + (D == 64 ? which * kGroupBytes : 0);
      const uint32_t acc = lane_base + cfg::o_col(n);
      const float* z = nullptr;  // NORM: what the other chunks add to this row, scaled by `scale`
      float scale = 1.f;
      if (NORM && which != 1) {
        z = (which == 0 ? p.zq : p.zk) + (static_cast<size_t>(bh) * n_iter + mem_chunk(n / 3)) * p.dim;
        const int tok = mem_chunk(n / 3) * kChunk + row;
        if (which == 2) scale = tok < p.n_tokens ? __ldg(p.d + static_cast<size_t>(bh) * p.n_tokens + tok) : 0.f;
      }
      // this warp's earlier stores have read the rows that are overwritten below (at D = 64 too all of them are
      // waited for, although each gradient has a stage of its own)
      if (lane == 0) ptx::bulk_wait_group_read0();
      __syncwarp();
      if (!wait_tmem(o_full(n), (n >> 1) & 1)) break;
#pragma unroll 1
      for (int gg = 0; gg < cfg::G; ++gg) {  // one 64-column group at a time, as registers allow
        ptx::tmem_ld32x2(acc + gg * 64, ra, acc + gg * 64 + 32, rb);
        const uint32_t dst = stage + gg * kGroupBytes + row * 128;
        auto store_half = [&](uint32_t j0, uint32_t (&r)[32]) {
          if (NORM && z != nullptr) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const int c = gg * 64 + static_cast<int>(j0) * 8 + j;  // dk is a multiple of 8
              float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
              if (c < p.dim) x = __ldg(reinterpret_cast<const float4*>(z + c));
              r[j] = __float_as_uint(__uint_as_float(r[j]) + scale * x.x);
              r[j + 1] = __float_as_uint(__uint_as_float(r[j + 1]) + scale * x.y);
              r[j + 2] = __float_as_uint(__uint_as_float(r[j + 2]) + scale * x.z);
              r[j + 3] = __float_as_uint(__uint_as_float(r[j + 3]) + scale * x.w);
            }
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            ptx::st_shared_v4(dst + (((j0 + j) ^ swz) << 4),
                              ptx::pack16x2<HALF>(__uint_as_float(r[8 * j + 0]), __uint_as_float(r[8 * j + 1])),
                              ptx::pack16x2<HALF>(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3])),
                              ptx::pack16x2<HALF>(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5])),
                              ptx::pack16x2<HALF>(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7])));
        };
        store_half(0, ra);
        store_half(4, rb);
      }
      // the accumulator may be overwritten (signalled after the loaded registers were used, see fla_kernel.cuh)
      ptx::tc_fence_before();
      ptx::mbar_arrive(o_free(n));
      ptx::fence_proxy_async_smem();
      __syncwarp();
      const int tok = mem_chunk(n / 3) * kChunk + quad * 32;
      if (lane == 0 && tok < p.n_tokens) {
#pragma unroll
        for (int gg = 0; gg < cfg::G; ++gg)
          ptx::tma_store_4d(map, stage + gg * kGroupBytes + quad * (32 * 128), gg * 64, tok, h, b);
        ptx::bulk_commit_group();
      }
    }
    if (lane == 0) ptx::bulk_wait_group0();
  } else {
    // ================================================================ converters of the states
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t swz = static_cast<uint32_t>(row & 7);
    // A state -> its 16-bit copy, [64-column group][row][128 B], 16-byte pieces XOR-swizzled by (row % 8).
    auto convert = [&](uint32_t state, uint32_t copy) {
      uint32_t r[32];
      if (quad * 32 < D) {
#pragma unroll 1
        for (int cb = 0; cb < D / 32; ++cb) {
          ptx::tmem_ld32(state + cb * 32, r);
          const uint32_t dst = copy + (cb >> 1) * (D * 128) + row * 128;
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            const uint32_t a0 = ptx::pack16x2<HALF>(__uint_as_float(r[jj * 8 + 0]), __uint_as_float(r[jj * 8 + 1]));
            const uint32_t a1 = ptx::pack16x2<HALF>(__uint_as_float(r[jj * 8 + 2]), __uint_as_float(r[jj * 8 + 3]));
            const uint32_t a2 = ptx::pack16x2<HALF>(__uint_as_float(r[jj * 8 + 4]), __uint_as_float(r[jj * 8 + 5]));
            const uint32_t a3 = ptx::pack16x2<HALF>(__uint_as_float(r[jj * 8 + 6]), __uint_as_float(r[jj * 8 + 7]));
            ptx::st_shared_v4(dst + ((((cb & 1) * 4 + jj) ^ swz) << 4), a0, a1, a2, a3);
          }
        }
      }
      ptx::fence_proxy_async_smem();
      ptx::tc_fence_before();
    };
    for (int i = 0; i < n_iter; ++i) {
      const bool last = i + 1 == n_iter;
      const bool to_final = last && p.r_final != nullptr;
      // S: its copy is free once dQ's first group of the last chunk is done, which this S being complete
      // implies (the groups were issued in that order)
      if (!wait_tmem(s_full, i & 1)) break;
      convert(lane_base + cfg::S_COL, sb_addr);
      ptx::mbar_arrive(sb_ready);
      // R: its copy is free once dV is complete. (The next completion of that o_full needs the rb_ready
      // below.)
      if (!last || to_final) {
        if (!wait_uniform(o_full(3 * i + 1), ((3 * i + 1) >> 1) & 1)) break;
        if (!wait_tmem(r_full, i & 1)) break;
        if (!last) {
          convert(lane_base + cfg::R_COL, rb_addr);
          ptx::mbar_arrive(rb_ready);
        } else {
          write_final_rows<D>(p.r_final + static_cast<size_t>(bh) * p.dim * p.dim, p.dim, lane_base + cfg::R_COL,
                              rb_addr + static_cast<uint32_t>(warp - 14) * 4096u, quad);
        }
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  __syncwarp();
  if (warp == 1) wait_uniform(drained, 0);
  if (*abort_flag) __nanosleep(100000);  // a wait gave up: let copies in flight land
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, cfg::TMEM_COLS);
  }
  if (threadIdx.x == 0 && *abort_flag && p.status != nullptr) atomicOr(p.status, 1);
}

}  // namespace fla
