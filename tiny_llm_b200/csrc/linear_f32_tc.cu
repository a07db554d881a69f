// float32 products C[M,N] = A[M,K] . W[N,K]^T on the 5th-generation tensor cores, for the 32-bit path: every factor is
// the sum of three bfloat16 values (24 bits of mantissa in three times 8: x = hi + mid + lo, each what is left rounded to
// nearest, so that mid is at most 2^-8 of x, lo 2^-17, and both have either sign), and a product is the sum of eight
// partial products: all but lo lo, which is below 2^-33 of it.  (Parts cut instead of rounded have the sign of x and up to
// twice the size; with them and six products a single product was up to 4.7e-7 off, an fmaf is 6.0e-8 at most.)
//
// The tensor cores cut what an fmaf rounds, so the accumulator of hi hi does not live long: after every 64 values of k
// it is read back, added to 32-bit sums in registers, and starts again from nothing.  The seven small products, 2^-8 of the
// whole and less, share accumulators that live through a slice of K and join its sum once: what is cut there is 2^-32.
// Relative error against 64 bits, 2-norm, normal operands, here / one chain of fmaf: K = 2,048 0.9e-7 to 1.3e-7 / 8.1e-7,
// K = 5,632 1.1e-7 / 1.3e-6.  Rows of few values (rms in sizes |a w| added up, 1 / 2 / 4 / 8 / 16 of 2,048 values): 2.5e-8, 2.1,
// 1.8, 1.4, 1.3e-8 in one slice of K, 2.6e-8, 3.0, 2.9, 2.5, 1.9e-8 in eight (a rounding more per slice), the chain 2.5e-8, 2.6,
// 2.7, 2.7, 2.9e-8.
//
// The sums' order is a function of N and K alone (`slices` must be one) -- k ascending in blocks of 64 within each of `slices` runs of blocks, the
// runs added in pairs, pairs of pairs and so on -- whatever M is and whichever shape of the kernel takes it, so a row's
// result does not depend on its batch, to the bit.
//
// Roles of a CTA, which makes 128 rows of W by BN rows of A over one slice of K:
//   a producer lane fetches 32 values of k of both as float32 (TMA, 128-byte swizzle);
//   warps that own a weight row per lane split it into tensor memory, the left operand of the MMAs;
//   warps that split the rows of A into shared memory, the right operand ([hi; mid; lo] below one another, K-major);
//   an MMA warp; and warps that own the running sums.
// The slices of a tile, or pairs of slices that a CTA walks one after the other, are a thread-block cluster that adds its sums
// through distributed shared memory.
//
// A sum that is not finite (an operand was infinite, NaN or above 2^104, or the sums above 2^80) is computed again as the
// other kernels of the 32-bit path compute every element, as one chain of fmaf: infinities and NaN come out as they do there.
//
// Takes whole boxes only: N a multiple of 32, K of 32, rows on 16 bytes.  Every wait is bounded (status word).
#include <cstdint>

#include "tc_common.cuh"

TLLM_DEFINE_LAST_ERROR

namespace tllm {

constexpr int ROWS = 128;            // weight rows per CTA = MMA M
constexpr int KS = 32;               // values of k per step: one 128-byte row of float32
constexpr int ROW_BYTES = 128;
constexpr int OUT_STORE = 1, OUT_ADD = 2;

template <int BN_, int RAW_, int STAGES_, int DBUF_, int W_GROUPS_, int T_GROUPS_, int T_WARPS_, int E_COLS_, int CTAS_,
          bool PAIRS_ = false, int REGS_ = 0>
struct Shape {
  static constexpr int BN = BN_;               // rows of A per CTA
  static constexpr int RAW = RAW_;             // steps of float32 in flight
  static constexpr int STAGES = STAGES_;       // split steps in flight
  static constexpr int DBUF = DBUF_;           // accumulators of hi hi
  static constexpr int W_GROUPS = W_GROUPS_;   // groups of four warps that split weights, step by step in turn
  static constexpr int T_GROUPS = T_GROUPS_, T_WARPS = T_WARPS_;   // groups of warps that split rows of A, in turn as well
  static constexpr int E_COLS = E_COLS_;       // columns per warp of the running sums
  static constexpr int CTAS = CTAS_;           // per SM
  static constexpr bool PAIRS = PAIRS_;        // may walk two slices
  static constexpr int REGS = REGS_;           // > 0: registers of a summing thread; the others give theirs up (whole warpgroups)
  static constexpr int S_READ = PAIRS || E_COLS > 16 ? 8 : 16;     // columns of small products read at a time (registers)
  static constexpr int E_WARPS = 4 * (BN / E_COLS);
  static constexpr int W0 = REGS > 0 ? 4 : 2, T0 = W0 + 4 * W_GROUPS, E0 = T0 + T_GROUPS * T_WARPS, WARPS = E0 + E_WARPS, THREADS = WARPS * 32;
  static constexpr int W_RAW = ROWS * ROW_BYTES, T_RAW = BN * ROW_BYTES, RAW_BYTES = W_RAW + T_RAW;
  static constexpr int B_SLOT = 3 * BN * ROW_BYTES;                // 64 values of k: the halves are neighbouring stages
  static constexpr int B_SLOTS = (STAGES + 1) / 2;
  static constexpr int B_OFFSET = RAW * RAW_BYTES;
  static constexpr int BAR_OFFSET = B_OFFSET + B_SLOTS * B_SLOT;
  static constexpr int BARS = 2 * RAW + 2 * STAGES + 2 * DBUF + 3;
  static constexpr int SMEM = BAR_OFFSET + BARS * 8 + 16 + 1024;   // + alignment slack
  // tensor memory: the small products' two accumulators, those of hi hi, split weight steps
  static constexpr int A_COLS = 3 * (KS / 2);
  static constexpr int D_BASE = 2 * BN, A_BASE = D_BASE + DBUF * BN;
  static constexpr int TMEM_USED = A_BASE + STAGES * A_COLS;
  static constexpr int TMEM_COLS = TMEM_USED <= 256 ? 256 : 512;
  // (a split of registers draws on what the block was launched with)
  static constexpr int LAUNCH_REGS = 65536 / THREADS / 8 * 8, OTHER_REGS = 48;
  static_assert(REGS == 0 || (E0 % 4 == 0 && E_WARPS % 4 == 0 && E_WARPS * 32 * REGS + E0 * 32 * OTHER_REGS <= THREADS * LAUNCH_REGS), "registers");
  static_assert(TMEM_USED <= 512 && CTAS * TMEM_COLS <= 512, "tensor memory");
  static_assert(2 * BN <= 256 && DBUF <= 2, "one MMA's columns; accumulators");
  static_assert(BN * ROWS * 4 <= B_OFFSET, "the sums are parked where the float32 steps were");
  static_assert(BN * (KS / 8) % (T_WARPS * 32) == 0, "whole tasks per lane");
  // A role waits by parity, so a slot's use before the one it waits for must not be two behind: either the slot's uses are
  // all its group's own, or the step it last did (which waited for the MMAs of STAGES steps before) lies late enough.
  static constexpr bool ordered(int slots, int groups) { return slots % groups == 0 || slots >= STAGES + groups; }
  static_assert(ordered(RAW, W_GROUPS) && ordered(RAW, T_GROUPS) && STAGES >= 2 && W_GROUPS <= 2 && T_GROUPS <= 2, "waits by parity");
};

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_ld8_issue(uint32_t taddr, uint32_t* r) {   // (tmem_ld_wait() before the values are used)
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ float4 ld_shared4(uint32_t at) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
  return v;
}
__device__ __forceinline__ void st_shared4(uint32_t at, const uint32_t* v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ float4 ld_peer4(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Two neighbouring values, times 2^24, as three pairs of bfloat16, the first of a pair in the low half.  All four subtractions
// are exact, and with the factor every float32 below 2^104 is the sum of its parts: without it the last part of a value below
// 2^-110 fell under bfloat16's smallest number (operands of 1e-35 gave products 5e-6 off, 2e-38 3e-3).  A larger value, or a sum
// of 2^80 and more, overflows, and the element is made as one chain of fmaf.
constexpr float SPLIT_SCALE = 16777216.f, SUM_SCALE = 1.f / (16777216.f * 16777216.f);
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  auto join = [](float a, float b) { uint64_t v; asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); return v; };
  auto round = [](uint64_t v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  };
  auto less = [&](uint64_t v, uint32_t part) {      // v - part
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(join(__uint_as_float(part << 16), __uint_as_float(part & 0xffff0000u))), "l"(join(-1.f, -1.f)), "l"(v));
    return r;
  };
  uint64_t v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(join(x, y)), "l"(join(SPLIT_SCALE, SPLIT_SCALE)));
  hi = round(v);
  v = less(v, hi);
  mid = round(v);
  lo = round(less(v, mid));
}

// One element as the other kernels of the 32-bit path make it.  NaN stays NaN, so the chain ends there: rows of NaN (a broken
// prompt's) cost a read each instead of K (11,264 x 2,048, 300 rows of NaN: 17,300 us -> 164, other rows
// 147; one NaN or infinity near a row's end, in pieces of 16 bytes: 17,300 -> 8,900).
__device__ __noinline__ float chain(const float* __restrict__ a, const float* __restrict__ w, int k) {
  float s = 0.f;
  for (int i = 0; i < k && !isnan(s); i += 4) {      // (rows on 16 bytes, K a multiple of 32)
    const float4 x = *reinterpret_cast<const float4*>(a + i), y = *reinterpret_cast<const float4*>(w + i);
    s = fmaf(x.x, y.x, s);
    s = fmaf(x.y, y.y, s);
    s = fmaf(x.z, y.z, s);
    s = fmaf(x.w, y.w, s);
  }
  return s;
}

template <typename S, int MODE>
__global__ void __launch_bounds__(S::THREADS, S::CTAS)
linear_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                     const float* __restrict__ a, const float* __restrict__ w, float* __restrict__ out, int m, int n, int k,
                     int lda, int ldo, int blocks_per_slice, int slices_per_cta, int early, int* __restrict__ status) {
  constexpr int BN = S::BN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + S::BAR_OFFSET);
  uint64_t* raw_empty = raw_full + S::RAW;
  uint64_t* split_full = raw_empty + S::RAW;
  uint64_t* split_empty = split_full + S::STAGES;
  uint64_t* d_full = split_empty + S::STAGES;      // [DBUF]: a block's hi hi lies in tensor memory / has been read
  uint64_t* d_empty = d_full + S::DBUF;
  uint64_t* s_full = d_empty + S::DBUF;            // a slice's small products lie in tensor memory / have been read
  uint64_t* s_empty = s_full + 1;
  uint64_t* end_bar = s_empty + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(end_bar + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * BN, n0 = blockIdx.y * ROWS;
  const int all_blocks = (k + 2 * KS - 1) / (2 * KS);
  const int block0 = blockIdx.z * slices_per_cta * blocks_per_slice;
  const int blocks = max(0, min(all_blocks - block0, slices_per_cta * blocks_per_slice));
  const int steps = 2 * blocks;                    // (an odd last step reads zeros past the end of K)
  const int k0 = block0 * 2 * KS;
  auto ends_slice = [&](int block) { return block == blocks - 1 || (S::PAIRS && block == blocks_per_slice - 1); };

  if (threadIdx.x == 0) {
    tma_prefetch_map(&map_w);
    tma_prefetch_map(&map_a);
    for (int s = 0; s < S::RAW; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], 4 + S::T_WARPS); }
    for (int s = 0; s < S::STAGES; ++s) { mbar_init(&split_full[s], 4 + S::T_WARPS); mbar_init(&split_empty[s], 1); }
    for (int s = 0; s < S::DBUF; ++s) { mbar_init(&d_full[s], 1); mbar_init(&d_empty[s], S::E_WARPS); }
    mbar_init(s_full, 1);
    mbar_init(s_empty, S::E_WARPS);
    mbar_init(end_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, S::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();

  const uint32_t base = smem_u32(smem);
  if (warp < S::E0) {
    if (S::REGS > 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::OTHER_REGS));
    if (warp == 0) {
      // ---------------- producer
      if (lane == 0) {
        const uint64_t once = l2_evict_first_policy();
        auto load_w = [&](int i) {
          mbar_expect_tx(&raw_full[i % S::RAW], S::RAW_BYTES);
          uint8_t* dst = smem + (i % S::RAW) * S::RAW_BYTES;
          if (early) tma_load_2d_hint(dst, &map_w, k0 + i * KS, n0, &raw_full[i % S::RAW], once);   // few rows of A: read once
          else tma_load_2d(dst, &map_w, k0 + i * KS, n0, &raw_full[i % S::RAW]);
        };
        auto load_a = [&](int i) {
          tma_load_2d(smem + (i % S::RAW) * S::RAW_BYTES + S::W_RAW, &map_a, k0 + i * KS, m0, &raw_full[i % S::RAW]);
        };
        const int pre = early ? min(steps, S::RAW) : 0;
        for (int i = 0; i < pre; ++i) load_w(i);
        pdl_wait();
        int i = 0;
        for (; i < steps; ++i) {
          if (i >= pre) {
            if (!mbar_wait(&raw_empty[i % S::RAW], ((i / S::RAW) & 1) ^ 1, abort_flag)) { *abort_flag = 1; atomicExch(status, ERR_FT_PRODUCER); break; }
            load_w(i);
          }
          load_a(i);
        }
        mbar_drain(raw_full, S::RAW, i);
      }
    } else if (warp == 1) {
      // ---------------- MMA issuer (the warp walks the loop converged, one lane issues)
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      const uint32_t b_lo0 = smem_desc_sw128_lo(base + S::B_OFFSET);
      constexpr uint32_t PART = (uint32_t)(BN * ROW_BYTES) >> 4;   // from hi to mid to lo, in descriptor units
      const uint32_t two = instr_desc_bf16(ROWS, 2 * BN), one = instr_desc_bf16(ROWS, BN);
      bool ok = true;
      for (int i = 0; i < steps; ++i) {
        const int s = i % S::STAGES, half = i & 1, block = i >> 1, set = block % S::DBUF;
        const bool second = S::PAIRS && half == 0 && block == blocks_per_slice, fresh = i == 0 || second;
        ok = mbar_wait(&split_full[s], (i / S::STAGES) & 1, abort_flag);
        if (second) ok = ok && mbar_wait(s_empty, 0, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t at = tm + S::A_BASE + s * S::A_COLS, d = tm + S::D_BASE + set * BN;
        const uint32_t bt = b_lo0 + (uint32_t)((s >> 1) * S::B_SLOT >> 4) + (uint32_t)((s & 1) * 64 >> 4);
        auto small = [&](int q) {
          umma_bf16_ts_lo(tm, at + q * 8, bt + PART + q * 2, two, fresh && q == 0 ? 0u : 1u);   // hi x [mid | lo]
          umma_bf16_ts_lo(tm, at + 16 + q * 8, bt + q * 2, two, 1u);                            // mid x [hi | mid]
          umma_bf16_ts_lo(tm, at + 32 + q * 8, bt + q * 2, two, 1u);                            // lo x [hi | mid]
          umma_bf16_ts_lo(tm, at + 16 + q * 8, bt + 2 * PART + q * 2, one, 1u);                 // mid x [lo]
        };
        auto large = [&](int q) { umma_bf16_ts_lo(d, at + q * 8, bt + q * 2, one, half > 0 || q > 0 ? 1u : 0u); };   // hi x [hi]
        // One accumulator of hi hi: the small products of a block's first half are made while it is read out.  Two: it has been
        // read by now, and one run of ten products is the faster (eight rows of A, us, two runs / one: 11,264 x 2,048 23.2 /
        // 22.3, 2,048 x 5,632 17.0 / 16.2, 2,048 x 2,048 8.6 / 8.3).
        const bool apart = S::DBUF == 1 && half == 0;
        if (apart) {
          if (elect_one()) { small(0); small(1); }
          __syncwarp();
        }
        if (half == 0) {
          ok = __all_sync(0xffffffffu, mbar_wait(&d_empty[set], ((block / S::DBUF) & 1) ^ 1, abort_flag));
          if (!ok) break;
          tc_fence_after();
        }
        if (elect_one()) {
          if (!apart) { large(0); small(0); large(1); small(1); }
          else { large(0); large(1); }
          umma_commit(&split_empty[s]);
          if (half == 1) umma_commit(&d_full[set]);
          if (half == 1 && ends_slice(block)) umma_commit(s_full);
        }
        __syncwarp();
      }
      if (!ok && lane == 0) { *abort_flag = 1; atomicExch(status, ERR_FT_MMA); }
      // nothing is in flight when the tensor memory goes back
      if (elect_one()) umma_commit(end_bar);
      __syncwarp();
      mbar_drain(end_bar, 1, 1);
    } else if (warp >= S::W0 && warp < S::T0) {
      // ---------------- weights: this lane owns a row; 32 values of float32 -> three times 16 columns of pairs
      const int group = (warp - S::W0) / 4, quad = warp & 3, row = quad * 32 + lane;
      const uint32_t row_at = base + row * ROW_BYTES, t_at = tmem + S::A_BASE + ((uint32_t)(quad * 32) << 16);
      bool ok = true;
      for (int i = group; i < steps; i += S::W_GROUPS) {
        const int r = i % S::RAW, s = i % S::STAGES;
        ok = mbar_wait(&raw_full[r], (i / S::RAW) & 1, abort_flag);
        ok = ok && mbar_wait(&split_empty[s], ((i / S::STAGES) & 1) ^ 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t src = row_at + r * S::RAW_BYTES, dst = t_at + s * S::A_COLS;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float4 v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = ld_shared4(src + (uint32_t)(((q * 4 + j) ^ (row & 7)) << 4));
          if (q == 1) {      // the float32 values are in registers
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_empty[r]);
          }
          uint32_t hi[8], mid[8], lo[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            split_pair(v[j].x, v[j].y, hi[2 * j], mid[2 * j], lo[2 * j]);
            split_pair(v[j].z, v[j].w, hi[2 * j + 1], mid[2 * j + 1], lo[2 * j + 1]);
          }
          tmem_st8(dst + q * 8, hi);
          tmem_st8(dst + 16 + q * 8, mid);
          tmem_st8(dst + 32 + q * 8, lo);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&split_full[s]);
      }
      if (!ok && lane == 0) { *abort_flag = 1; atomicExch(status, ERR_FT_SPLIT); }
    } else if (warp >= S::T0) {
      // ---------------- rows of A: eight values of a row per task, 16 bytes into each of the three tiles
      const int group = (warp - S::T0) / S::T_WARPS, t = (warp - S::T0) % S::T_WARPS * 32 + lane;
      constexpr int TASKS = BN * (KS / 8) / (S::T_WARPS * 32);
      bool ok = true;
      for (int i = group; i < steps; i += S::T_GROUPS) {
        const int r = i % S::RAW, s = i % S::STAGES;
        ok = mbar_wait(&raw_full[r], (i / S::RAW) & 1, abort_flag);
        ok = ok && mbar_wait(&split_empty[s], ((i / S::STAGES) & 1) ^ 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t src = base + r * S::RAW_BYTES + S::W_RAW, dst = base + S::B_OFFSET + (s >> 1) * S::B_SLOT;
#pragma unroll
        for (int j = 0; j < TASKS; ++j) {
          const int task = j * S::T_WARPS * 32 + t, row = task % BN, piece = task / BN;
          const float4 u = ld_shared4(src + row * ROW_BYTES + (uint32_t)(((2 * piece) ^ (row & 7)) << 4));
          const float4 v = ld_shared4(src + row * ROW_BYTES + (uint32_t)(((2 * piece + 1) ^ (row & 7)) << 4));
          uint32_t hi[4], mid[4], lo[4];
          split_pair(u.x, u.y, hi[0], mid[0], lo[0]);
          split_pair(u.z, u.w, hi[1], mid[1], lo[1]);
          split_pair(v.x, v.y, hi[2], mid[2], lo[2]);
          split_pair(v.z, v.w, hi[3], mid[3], lo[3]);
          const uint32_t to = dst + row * ROW_BYTES + (uint32_t)((((s & 1) * 4 + piece) ^ (row & 7)) << 4);
          st_shared4(to, hi);
          st_shared4(to + BN * ROW_BYTES, mid);
          st_shared4(to + 2 * BN * ROW_BYTES, lo);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) { mbar_arrive(&raw_empty[r]); mbar_arrive(&split_full[s]); }
      }
      if (!ok && lane == 0) { *abort_flag = 1; atomicExch(status, ERR_FT_SPLIT); }
    }
  } else {
    if (S::REGS > 0) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(S::REGS > 0 ? S::REGS : 232));
    // ---------------- running sums: this thread owns weight row `row` and E_COLS rows of A
    const int quad = warp & 3, row = quad * 32 + lane, c0 = (warp - S::E0) / 4 * S::E_COLS;
    const uint32_t t_at = tmem + ((uint32_t)(quad * 32) << 16) + c0;
    float acc[S::E_COLS], first[S::PAIRS ? S::E_COLS : 1];      // first: the first slice's sums, of two
#pragma unroll
    for (int c = 0; c < S::E_COLS; ++c) acc[c] = 0.f;
    if (S::PAIRS) {
#pragma unroll
      for (int c = 0; c < S::E_COLS; ++c) first[S::PAIRS ? c : 0] = 0.f;
    }
    bool ok = true;
    for (int b = 0; b < blocks && ok; ++b) {
      if (S::PAIRS && b == blocks_per_slice) {
#pragma unroll
        for (int c = 0; c < S::E_COLS; ++c) { first[S::PAIRS ? c : 0] = acc[c]; acc[c] = 0.f; }
      }
      const int set = b % S::DBUF;
      ok = __all_sync(0xffffffffu, mbar_wait(&d_full[set], (b / S::DBUF) & 1, abort_flag));
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < S::E_COLS; c += 16) {
        float v[16];
        tmem_ld16(t_at + S::D_BASE + set * BN + c, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[c + j] += v[j];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&d_empty[set]);
      if (ends_slice(b)) {
        ok = __all_sync(0xffffffffu, mbar_wait(s_full, b >= blocks_per_slice ? 1 : 0, abort_flag));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < S::E_COLS; c += S::S_READ) {
          uint32_t u[S::S_READ], v[S::S_READ];
#pragma unroll
          for (int j = 0; j < S::S_READ; j += 8) { tmem_ld8_issue(t_at + c + j, u + j); tmem_ld8_issue(t_at + BN + c + j, v + j); }
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < S::S_READ; ++j) acc[c + j] += __uint_as_float(u[j]) + __uint_as_float(v[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_empty);
      }
    }
    if (!ok && lane == 0) { *abort_flag = 1; atomicExch(status, ERR_FT_SUMS); }
    if (S::PAIRS && slices_per_cta == 2) {
      const bool one = blocks <= blocks_per_slice;     // (the second slice is empty: its sums are zeros)
#pragma unroll
      for (int c = 0; c < S::E_COLS; ++c) acc[c] = one ? acc[c] + 0.f : first[S::PAIRS ? c : 0] + acc[c];
    }
    // every step has been split by now (its MMAs are done): the float32 steps' place is free
    float* parked = reinterpret_cast<float*>(smem);     // [BN][128]
#pragma unroll
    for (int c = 0; c < S::E_COLS; ++c) parked[(c0 + c) * ROWS + row] = ok ? acc[c] : 0.f;
  }
  pdl_wait();     // (all threads: the output may be what an earlier launch still reads)
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, S::TMEM_COLS);

  // ---------------- the slices' sums, added in pairs; work items are four consecutive weight rows of one row of A
  cluster_sync();
  const int peers = gridDim.z, rows_per = ((ROWS + peers - 1) / peers + 3) & ~3, r0 = blockIdx.z * rows_per, quads = rows_per / 4;
  for (int idx = threadIdx.x; idx < quads * BN; idx += S::THREADS) {
    const int j = idx / quads, r = r0 + (idx % quads) * 4, gm = m0 + j, gn = n0 + r;
    if (gm >= m || r >= ROWS || gn >= n) continue;     // (N is a multiple of 32: four rows exist together)
    // missing slices are zeros; pairs that a smaller cluster's CTAs have walked are the same pairs
    float4 part[8];
#pragma unroll
    for (int z = 0; z < 8; ++z)
      part[z] = z < peers ? ld_peer4(base + (uint32_t)(j * ROWS + r) * 4u, z) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int d = 1; d < 8; d *= 2)
#pragma unroll
      for (int z = 0; z + d < 8; z += 2 * d) {
        part[z].x += part[z + d].x; part[z].y += part[z + d].y; part[z].z += part[z + d].z; part[z].w += part[z + d].w;
      }
    float sum[4] = {part[0].x, part[0].y, part[0].z, part[0].w};
    float* dst = out + (size_t)gm * ldo + gn;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      sum[e] = isfinite(sum[e]) ? sum[e] * SUM_SCALE : chain(a + (size_t)gm * lda, w + (size_t)(gn + e) * k, k);
      if (MODE == OUT_ADD) dst[e] += sum[e];
      else dst[e] = sum[e];
    }
  }
  cluster_sync();   // no CTA leaves while a peer still reads its shared memory
}

// ---------------------------------------------------------------- host side
// A float32 matrix [rows, k] with row stride ld, in boxes of `box` rows x 32 values.
static bool make_f32_map(CUtensorMap* map, const float* ptr, int rows, int k, long long ld, int box) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t boxes[2] = {(cuuint32_t)KS, (cuuint32_t)box};
  cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, boxes, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename S, int MODE>
static int launch_mode(const float* a, const float* w, float* out, int m, int n, int k, int lda, int ldo, int slices, int early,
                       int* status, cudaStream_t s, int sms) {
  auto kern = linear_f32_tc_kernel<S, MODE>;
  TLLM_RESERVE_SMEM("linear_f32_tc", S::SMEM, kern);
  CUtensorMap mw, ma;
  if (!make_f32_map(&mw, w, n, k, k, ROWS) || !make_f32_map(&ma, a, m, k, lda, S::BN))
    TLLM_FAIL(TLLM_ERR_CUDA, "linear_f32_tc: cuTensorMapEncodeTiled failed");
  const int blocks = (k + 2 * KS - 1) / (2 * KS), per = (blocks + slices - 1) / slices;
  const int tiles_m = (m + S::BN - 1) / S::BN, tiles_n = (n + ROWS - 1) / ROWS;
  // Two slices per CTA where one each are more CTAs than SMs: what a CTA pays once, its first steps' way from memory and its
  // sums' way out, comes half as often.  (us, eight CTAs of one slice / four of two: 509 rows, 2,560 x 2,048 92 / 63, 2,048 x
  // 2,048 76 / 43, 2,048 x 5,632 130 / 86; 131 rows, 2,048 x 2,048 39 / 21.)
  const int each = S::PAIRS && slices > 2 && (long long)tiles_m * tiles_n * slices > sms ? 2 : 1, ctas = (slices + each - 1) / each;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles_m, tiles_n, ctas);
  cfg.blockDim = dim3(S::THREADS);
  cfg.dynamicSmemBytes = S::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = ctas;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, mw, ma, a, w, out, m, n, k, lda, ldo, per, each, early, status);
  if (e != cudaSuccess) TLLM_FAIL(TLLM_ERR_CUDA, "linear_f32_tc: %s", cudaGetErrorString(e));
  return TLLM_OK;
}

template <typename S>
static int launch_shape(const float* a, const float* w, float* out, int m, int n, int k, int lda, int ldo, int mode, int slices,
                        int early, int* status, cudaStream_t s, int sms) {
  if (mode == OUT_ADD) return launch_mode<S, OUT_ADD>(a, w, out, m, n, k, lda, ldo, slices, early, status, s, sms);
  return launch_mode<S, OUT_STORE>(a, w, out, m, n, k, lda, ldo, slices, early, status, s, sms);
}

// Which shape: the smallest that holds the rows.  Few rows are bound by the weights from memory, up to 6 TB/s of them with two
// CTAs on every SM, and by what a launch takes whatever it multiplies (7.8 us for 2,048 x 2,048, whose weights take 2.6); many by
// the tensor cores and the read-out beside them.  us, m = 1 / 8 / 64 / 509, launches in a graph, weights from memory, one chain of
// fmaf per element: 2,560 x 2,048 7.8 / 13.4 / 55 / 144, 2,048 x 2,048 7.5 / 12.9 / 37 / 101, 11,264 x 2,048 23.1 / 27.3 / 103 /
// 458, 2,048 x 5,632 18.6 / 33.6 / 99 / 274; here 8.2 / 8.5 / 15.4 / 63, 7.8 / 8.3 / 20.8 / 43, 22.1 / 22.4 / 48 / 166, 15.7 /
// 16.3 / 36 / 86.  With six products and parts that are cut: 8.2 / 8.6 / 14.7 / 64, 8.1 / 8.4 / 20.6 / 43, 21.9 / 22.3 / 46 / 174,
// 16.0 / 16.3 / 35 / 89: the two products more cost 33 to 64 rows 1 to 6 %.  (Without the factor of split_pair 11,264 x 2,048 took
// 162 instead of 166 for 509 rows, few rows the same; with scalar multiplications and subtractions instead of pairs eight rows took 23.5
// and 17.8 for the two large ones.)
// Other forms of Shape64: weights split by two groups of warps 2 to 3 % slower, three or four stages 1 to 4 %.
//                    BN RAW STAGES DBUF W_GROUPS T_GROUPS T_WARPS E_COLS CTAS PAIRS REGS
using Shape16 = Shape<16, 5, 3, 2, 2, 2, 1, 16, 2>;
using Shape128 = Shape<128, 5, 2, 1, 1, 1, 4, 64, 1, true, 168>;
using Shape32 = Shape<32, 4, 2, 2, 2, 1, 2, 32, 2>;
using Shape64 = Shape<64, 6, 2, 2, 1, 1, 4, 32, 1, true>;

}  // namespace tllm

using namespace tllm;

// out[M, N] (float32, row stride ldo) = / += a[M, K] (row stride lda) . w[N, K]^T; mode 1 store, 2 add.  `slices` of K (1 to
// 8) must depend on N and K alone.  At most 16 rows: the weights are read ahead of the launches before, which therefore may
// not be writing them.
extern "C" int tllm_linear_f32_tc(const void* a, const void* w, void* out, int m, int n, int k, int lda, int ldo, int mode,
                                  int slices, int* status, void* stream) {
  TLLM_REQUIRE(m > 0 && n > 0 && k > 0, "linear_f32_tc: empty product %d x %d x %d", m, n, k);
  TLLM_REQUIRE(n % 32 == 0 && k % 32 == 0 && lda % 4 == 0 && lda >= k && ldo >= n, "linear_f32_tc: %d x %d weights, row strides %d and %d (multiples of 32, rows on 16 bytes)", n, k, lda, ldo);
  TLLM_REQUIRE(((uintptr_t)a % 16) == 0 && ((uintptr_t)w % 16) == 0, "linear_f32_tc: operands must be 16-byte aligned");
  TLLM_REQUIRE(slices >= 1 && slices <= 8 && slices <= (k + 63) / 64, "linear_f32_tc: %d slices of a K of %d", slices, k);
  TLLM_REQUIRE((mode == OUT_STORE || mode == OUT_ADD) && status != nullptr, "linear_f32_tc: mode %d", mode);
  TLLM_REQUIRE((n + ROWS - 1) / ROWS <= 65535, "linear_f32_tc: %d weight rows exceed the grid", n);
  const float* af = (const float*)a;
  const float* wf = (const float*)w;
  float* of = (float*)out;
  cudaStream_t s = (cudaStream_t)stream;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    TLLM_FAIL(TLLM_ERR_CUDA, "linear_f32_tc: cannot read the number of SMs");
  if (m <= 16) return launch_shape<Shape16>(af, wf, of, m, n, k, lda, ldo, mode, slices, 1, status, s, sms);
  if (m <= 32) return launch_shape<Shape32>(af, wf, of, m, n, k, lda, ldo, mode, slices, 0, status, s, sms);
  if (m <= 64) return launch_shape<Shape64>(af, wf, of, m, n, k, lda, ldo, mode, slices, 0, status, s, sms);
  return launch_shape<Shape128>(af, wf, of, m, n, k, lda, ldo, mode, slices, 0, status, s, sms);
}
