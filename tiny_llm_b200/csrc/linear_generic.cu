// C[M,N] = A[M,K] . W[N,K]^T on the CUDA cores with 32-bit accumulation (FFMA only, no tensor-core
// mode): the products of the 32-bit path that linear_f32_tc.cu does not take, and the fallback of the bfloat16 path for sizes the
// tensor-core kernels refuse.  Any M, N, K.  Every output element is ONE chain of fmaf over k in
// ascending order starting from zero, whatever M is and whichever of the kernels below computes it,
// so a row's result does not depend on its batch, to the bit.
//   linear_generic_kernel: 64 x 64 tiles, 4 x 4 outputs per thread (any sizes and both dtypes);
//   linear_tiled_kernel: float32, more than 16 rows, rows on 16 bytes: tiles from 16 x 64 to 64 x 192 by the sizes;
//   linear_skinny_kernel: float32, at most 16 rows (decoded tokens), rows on 16 bytes: the weights stream through a ring
//     of TMA boxes.
// A bounded wait that runs out leaves a code in the device's status word.
// Reference counterpart: tiny_llm/ops/cuda/gemm.cu:67-106 (64x256 tile, 8x8 outputs per thread).
#include <cstdint>

#include "tc_common.cuh"

TLLM_DEFINE_LAST_ERROR

namespace tllm {

constexpr int BM = 64, BN = 64, BK = 16, THREADS = 256;

// out modes
constexpr int OUT_SAME = 0;   // store in the input dtype
constexpr int OUT_F32 = 1;    // store float32
constexpr int OUT_ACC = 2;    // out (float32) += product

template <typename T, int MODE>
__global__ void __launch_bounds__(THREADS)
linear_generic_kernel(const T* __restrict__ a, const T* __restrict__ w, void* __restrict__ out,
                      int m, int n, int k, int lda, int ldo) {
  __shared__ float as[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int lk = tid % BK, lr = tid / BK;  // loader: k index and first row; rows lr + 16 i
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < k; k0 += BK) {
    const int kk = k0 + lk;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = lr + 16 * i;
      const int gm = m0 + r, gn = n0 + r;
      as[lk][r] = (gm < m && kk < k) ? to_f32(a[(size_t)gm * lda + kk]) : 0.f;
      ws[lk][r] = (gn < n && kk < k) ? to_f32(w[(size_t)gn * k + kk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < BK; ++p) {
      const float4 av = *reinterpret_cast<const float4*>(&as[p][ty * 4]);
      const float4 wv = *reinterpret_cast<const float4*>(&ws[p][tx * 4]);
      const float ar[4] = {av.x, av.y, av.z, av.w};
      const float wr[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ar[i], wr[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty * 4 + i;
    if (gm >= m) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn >= n) continue;
      const size_t o = (size_t)gm * ldo + gn;
      if (MODE == OUT_SAME) reinterpret_cast<T*>(out)[o] = from_f32<T>(acc[i][j]);
      else if (MODE == OUT_F32) reinterpret_cast<float*>(out)[o] = acc[i][j];
      else reinterpret_cast<float*>(out)[o] += acc[i][j];
    }
  }
}

// ---------------------------------------------------------------- more than 16 rows, float32: tiles of fma pairs
// The same chains of fmaf (k ascending from zero for every output element; fma.rn.f32x2 rounds each half like fmaf).
// What bounds it: the fma pipe.  A packed fma keeps the pipe busy for two cycles with one issue slot, which leaves the
// other slot for the operands; a thread's outputs are pairs of neighbouring columns, so that a pair of weights is one
// half of a 16-byte read and only the row's value has to be doubled in a register.
// Two producer warps beside the computing ones keep cp.async copies of the next TST steps of TBK values of k in flight
// (a step of products is shorter than a trip to memory: with one step of look-ahead in registers a CTA alone on an SM
// took 182 cycles per k for 128 x 128 outputs) and turn each landed step into [k][row] order, from which a computing
// thread reads four rows or four columns at once, while the step before is multiplied: one barrier per step.
// Measured on 509 x 2,048 x 2,048 / 509 x 11,264 x 2,048 / 509 x 2,048 x 5,632, us: 128 x 128 tiles of single fmaf with
// register look-ahead 239 / 697 / 638; these tiles 102 / 457 / 269 (the pipe's own time: 57 / 316 / 158).
__device__ __forceinline__ uint64_t pack_pair(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_pair(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// 16 bytes on their way to shared memory; ok = false fills them with zeros, which leave a chain of fmaf as it is
__device__ __forceinline__ void copy16_async(uint32_t dst, const float* src, bool ok) {
  const int bytes = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

constexpr int TBK = 16, TST = 4, TPRODUCERS = 64;

// WM x WN computing warps, each (4 TM) x (8 TN) outputs, a thread TM x TN
template <int WM, int WN, int TM, int TN>
struct Tile {
  static constexpr int M = WM * 4 * TM, N = WN * 8 * TN, COMPUTE = WM * WN * 32, THREADS = COMPUTE + TPRODUCERS;
  static constexpr int PM = M + 4, PN = N + 4;                 // pitches of the [k][row] tiles
  static constexpr int RAW = (M + N) * TBK;                    // floats of a landed step: rows of A, then rows of W
  static constexpr int SMEM = (TST * RAW + 2 * TBK * (PM + PN)) * (int)sizeof(float);
  static constexpr int SMEM_ALONE = 120000;                    // more than half of an SM's: one CTA per SM
};

template <int WM, int WN, int TM, int TN, int MODE>
__global__ void __launch_bounds__((Tile<WM, WN, TM, TN>::THREADS), (TM * TN > 64 ? 1 : 2))
linear_tiled_kernel(const float* __restrict__ a, const float* __restrict__ w, float* __restrict__ out,
                    int m, int n, int k, int lda, int ldo) {
  using C = Tile<WM, WN, TM, TN>;
  constexpr int PM = C::PM, PN = C::PN, QK = TBK / 4;
  constexpr int LA = C::M * QK / TPRODUCERS, LW = C::N * QK / TPRODUCERS;   // 16-byte copies per producer and step
  static_assert(LA * TPRODUCERS == C::M * QK && LW * TPRODUCERS == C::N * QK, "whole copies per producer");
  extern __shared__ __align__(16) float tile_smem[];
  float* raw = tile_smem;
  float* as = tile_smem + TST * C::RAW;       // [2][TBK][PM]
  float* ws = as + 2 * TBK * PM;              // [2][TBK][PN]
  pdl_trigger();
  const int tid = threadIdx.x;
  const int m0 = blockIdx.x * C::M, n0 = blockIdx.y * C::N;
  const int steps = (k + TBK - 1) / TBK;

  if (tid >= C::COMPUTE) {
    // ---------------- producers
    const int pt = tid - C::COMPUTE;
    const uint32_t raw_u = (uint32_t)__cvta_generic_to_shared(raw);
    auto copy_w = [&](int st) {
      if (st >= steps) return;
      const uint32_t d = raw_u + (uint32_t)((st % TST) * C::RAW + C::M * TBK) * 4u;
#pragma unroll
      for (int i = 0; i < LW; ++i) {
        const int idx = pt + i * TPRODUCERS, r = n0 + idx / QK, kk = st * TBK + (idx % QK) * 4;   // k is a multiple of 4
        const bool ok = r < n && kk < k;
        copy16_async(d + idx * 16, ok ? w + (size_t)r * k + kk : w, ok);
      }
    };
    auto copy_a = [&](int st) {
      if (st >= steps) return;
      const uint32_t d = raw_u + (uint32_t)((st % TST) * C::RAW) * 4u;
#pragma unroll
      for (int i = 0; i < LA; ++i) {
        const int idx = pt + i * TPRODUCERS, r = m0 + idx / QK, kk = st * TBK + (idx % QK) * 4;
        const bool ok = r < m && kk < k;
        copy16_async(d + idx * 16, ok ? a + (size_t)r * lda + kk : a, ok);
      }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    pdl_wait();   // before the weights too: with this many rows `w` may be what the launch just before has written
    for (int st = 0; st < TST; ++st) { copy_w(st); copy_a(st); commit(); }
    for (int st = 0; st < steps; ++st) {
      asm volatile("cp.async.wait_group %0;" ::"n"(TST - 1) : "memory");
      // a producer turns what it copied itself, so its own landed groups are all it has to wait for
      const float4* rs = reinterpret_cast<const float4*>(raw + (st % TST) * C::RAW);
      float* ad = as + (st & 1) * TBK * PM;
      float* wd = ws + (st & 1) * TBK * PN;
#pragma unroll
      for (int i = 0; i < LA; ++i) {
        const int idx = pt + i * TPRODUCERS, r = idx / QK, q = (idx % QK) * 4;
        const float4 v = rs[idx];
        ad[q * PM + r] = v.x; ad[(q + 1) * PM + r] = v.y; ad[(q + 2) * PM + r] = v.z; ad[(q + 3) * PM + r] = v.w;
      }
#pragma unroll
      for (int i = 0; i < LW; ++i) {
        const int idx = pt + i * TPRODUCERS, r = idx / QK, q = (idx % QK) * 4;
        const float4 v = rs[C::M * QK + idx];
        wd[q * PN + r] = v.x; wd[(q + 1) * PN + r] = v.y; wd[(q + 2) * PN + r] = v.z; wd[(q + 3) * PN + r] = v.w;
      }
      copy_w(st + TST);
      copy_a(st + TST);
      commit();
      __syncthreads();   // step st can be read; everyone has left step st - 1, whose place step st + 1 takes
    }
    return;
  }

  // ---------------- computing warps
  pdl_wait();
  const int warp = tid >> 5, lane = tid & 31;
  const int ar0 = (warp / WN) * 4 * TM + (lane / 8) * 4;   // this thread's rows: ar0 + 16 i + {0..3}
  const int bc0 = (warp % WN) * 8 * TN + (lane % 8) * 4;   // ... and columns: bc0 + 32 j + {0..3}
  uint64_t acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
#pragma unroll 1
  for (int st = 0; st < steps; ++st) {
    __syncthreads();
    const float* ab = as + (st & 1) * TBK * PM + ar0;
    const float* wb = ws + (st & 1) * TBK * PN + bc0;
#pragma unroll
    for (int p = 0; p < TBK; ++p) {
      float4 a4[TM / 4];
      ulonglong2 w4[TN / 4];
#pragma unroll
      for (int i = 0; i < TM / 4; ++i) a4[i] = *reinterpret_cast<const float4*>(ab + p * PM + 16 * i);
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) w4[j] = *reinterpret_cast<const ulonglong2*>(wb + p * PN + 32 * j);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float av = (i & 3) == 0 ? a4[i / 4].x : (i & 3) == 1 ? a4[i / 4].y : (i & 3) == 2 ? a4[i / 4].z : a4[i / 4].w;
        const uint64_t aa = pack_pair(av, av);
#pragma unroll
        for (int j = 0; j < TN / 4; ++j) {
          acc[i][2 * j] = fma_pair(aa, w4[j].x, acc[i][2 * j]);
          acc[i][2 * j + 1] = fma_pair(aa, w4[j].y, acc[i][2 * j + 1]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ar0 + 16 * (i / 4) + (i & 3);
    if (gm >= m) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + bc0 + 32 * (j / 4) + (j & 3);
      if (gn >= n) continue;
      float lo, hi;
      unpack_pair(acc[i][j / 2], lo, hi);
      const float v = (j & 1) ? hi : lo;
      const size_t o = (size_t)gm * ldo + gn;
      if (MODE == OUT_ACC) out[o] += v;
      else out[o] = v;
    }
  }
}

template <int WM, int WN, int TM, int TN, int MODE>
static int launch_tile_mode(const float* a, const float* w, float* out, int m, int n, int k, int lda, int ldo, int sms, cudaStream_t s) {
  using C = Tile<WM, WN, TM, TN>;
  auto kern = linear_tiled_kernel<WM, WN, TM, TN, MODE>;
  constexpr int MOST = C::SMEM > C::SMEM_ALONE ? C::SMEM : C::SMEM_ALONE;
  TLLM_RESERVE_SMEM("linear_tiled", MOST, kern);
  dim3 grid((m + C::M - 1) / C::M, (n + C::N - 1) / C::N);
  // As many CTAs as SMs or fewer: one per SM.  Two that may share an SM do so while others idle (128 CTAs of 64 x 128
  // took 155 us instead of 102).
  const int smem = (long long)grid.x * grid.y <= sms ? MOST : C::SMEM;
  TLLM_LAUNCH("linear_tiled", kern, grid, C::THREADS, smem, s, a, w, out, m, n, k, lda, ldo);
  return TLLM_OK;
}

template <int WM, int WN, int TM, int TN>
static int launch_tile(const float* a, const float* w, float* out, int m, int n, int k, int lda, int ldo, int mode, int sms, cudaStream_t s) {
  if (mode == OUT_ACC) return launch_tile_mode<WM, WN, TM, TN, OUT_ACC>(a, w, out, m, n, k, lda, ldo, sms, s);
  return launch_tile_mode<WM, WN, TM, TN, OUT_F32>(a, w, out, m, n, k, lda, ldo, sms, s);
}

// Which tile: the one whose rounds over the SMs cost least, with the measured cycles per k of a tile alone on an SM.
// (m x n x k, us, chosen against the other tiles: 509 x 2,560 x 2,048 64 x 192 147 / 64 x 128 193; 200 x 2,560 64 x 128
// 100 / 64 x 64 128; 100 x 2,560 64 x 64 73 / 64 x 128 100; 100 x 2,048 x 5,632 32 x 64 152 / 64 x 64 193;
// 40 x 2,560 16 x 64 39 / 32 x 64 57; 40 x 11,264 64 x 128 100 / 16 x 64 135.)
static int launch_tiled(const float* a, const float* w, float* out, int m, int n, int k, int lda, int ldo, int mode, cudaStream_t s) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    TLLM_FAIL(TLLM_ERR_CUDA, "linear: cannot read the number of SMs");
  static const struct { int m, n, cycles; } kinds[] = {{64, 128, 95}, {64, 192, 137}, {64, 64, 70}, {32, 64, 54}, {16, 64, 37}};
  int best = 0;
  long long best_cost = -1;
  for (int i = 0; i < 5; ++i) {
    const long long ctas = (long long)((m + kinds[i].m - 1) / kinds[i].m) * ((n + kinds[i].n - 1) / kinds[i].n);
    const long long cost = (ctas + sms - 1) / sms * kinds[i].cycles;
    if (best_cost < 0 || cost < best_cost) { best = i; best_cost = cost; }
  }
  switch (best) {
    case 0: return launch_tile<2, 2, 8, 8>(a, w, out, m, n, k, lda, ldo, mode, sms, s);
    case 1: return launch_tile<2, 2, 8, 12>(a, w, out, m, n, k, lda, ldo, mode, sms, s);
    case 2: return launch_tile<2, 2, 8, 4>(a, w, out, m, n, k, lda, ldo, mode, sms, s);
    case 3: return launch_tile<2, 2, 4, 4>(a, w, out, m, n, k, lda, ldo, mode, sms, s);
    default: return launch_tile<1, 2, 4, 4>(a, w, out, m, n, k, lda, ldo, mode, sms, s);
  }
}

// ---------------------------------------------------------------- at most 16 rows, float32
// A CTA streams ROWS = W x RW weight rows and the R rows of A through a ring of TMA boxes of 32 k (128-byte swizzle: rows
// lie 128 bytes apart and 16-byte reads of eight rows do not collide), KB boxes per stage; a producer warp issues them,
// the weights' first stages before the wait for earlier kernels.  A lane owns one weight row and TR rows of A: TR chains of
// fmaf, whose operands it reads KS steps of four k ahead (read where they are used, every step stood behind a trip to
// shared memory).  What bounds it: the weights from memory where there are many rows of them, else the latencies of the few
// warps that an SM has (8 x 2,048 x 5,632: 3.3 warps, issue slots 16 % used, the load/store pipe 12 %; 8 x 11,264 x 2,048:
// 6.7, 26 and 19 %); the chains themselves (4 cycles per k) would take 4.3 us at K = 2,048.
// us, this kernel / one chain per thread with cp.async by the computing threads (m = 8): 2,560 x 2,048 14.9 / 26.8,
// 2,048 x 2,048 13.8 / 20.2, 11,264 x 2,048 27.4 / 43.5, 2,048 x 5,632 34.2 / 55.0, 32,000 x 2,048 74.6 / 115.7; m = 1:
// 9.0 / 18.3, 8.5 / 17.4, 23.8 / 26.9, 19.9 / 43.2, 46.9 / 50.0.
__device__ __forceinline__ float4 read_shared4(uint32_t at) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
  return v;
}

template <int R, int RW, int TR, int W, int KB, int ST>
struct Skinny {
  static constexpr int ROWS = W * RW, GROUPS = R / TR, KC = KB * 32;
  static_assert(GROUPS * TR == R && GROUPS * RW <= 32 && ROWS % 8 == 0, "lanes of a warp; whole swizzle atoms");
  static constexpr int W_BOX = ROWS * 128, A_BOX = R * 128, A_STEP = A_BOX < 1024 ? 1024 : A_BOX;
  static constexpr int STAGE = KB * (W_BOX + A_STEP);
  static constexpr int SMEM = ST * STAGE + 2 * ST * 8 + 16 + 1024;   // + alignment slack
};

template <int R, int RW, int TR, int W, int KB, int ST, int MODE>
__global__ void __launch_bounds__(W * 32 + 32)
linear_skinny_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                     float* __restrict__ out, int m, int n, int k, int ldo, int* __restrict__ status) {
  using C = Skinny<R, RW, TR, W, KB, ST>;
  extern __shared__ uint8_t sk_smem[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sk_smem) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + ST * C::STAGE);
  uint64_t* empty = full + ST;
  volatile uint32_t* abort_flag = reinterpret_cast<uint32_t*>(empty + ST);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n0 = blockIdx.x * C::ROWS, m0 = blockIdx.y * R;
  const int chunks = (k + C::KC - 1) / C::KC;
  if (tid == 0) {
    tma_prefetch_map(&map_w);
    tma_prefetch_map(&map_a);
    for (int s = 0; s < ST; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], W); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_trigger();

  if (warp == W) {
    // ---------------- producer
    if (lane == 0) {
      auto load_w = [&](int c) {
        const int s = c % ST;
        mbar_expect_tx(&full[s], KB * (C::W_BOX + C::A_BOX));
#pragma unroll
        for (int b = 0; b < KB; ++b) tma_load_2d(sm + s * C::STAGE + b * C::W_BOX, &map_w, c * C::KC + b * 32, n0, &full[s]);
      };
      auto load_a = [&](int c) {
        const int s = c % ST;
#pragma unroll
        for (int b = 0; b < KB; ++b)
          tma_load_2d(sm + s * C::STAGE + KB * C::W_BOX + b * C::A_STEP, &map_a, c * C::KC + b * 32, m0, &full[s]);
      };
      const int pre = min(chunks, ST);
      for (int c = 0; c < pre; ++c) load_w(c);
      pdl_wait();
      for (int c = 0; c < pre; ++c) load_a(c);
      int c = pre;
      for (; c < chunks; ++c) {
        if (!mbar_wait(&empty[c % ST], ((c / ST) & 1) ^ 1, abort_flag)) { *abort_flag = 1; atomicExch(status, ERR_SK_PRODUCER); break; }
        load_w(c);
        load_a(c);
      }
      mbar_drain(full, ST, c);
    }
    return;
  }

  // ---------------- computing warps
  pdl_wait();
  const bool computes = lane < RW * C::GROUPS;
  const int row = warp * RW + lane % RW, group = computes ? lane / RW : 0;   // weight row; rows of A group * TR + i
  uint32_t w_at[8], a_at[TR][8];                                             // 16-byte pieces of a box, unswizzled
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    w_at[j] = (uint32_t)(row * 128 + ((j ^ (row & 7)) << 4));
#pragma unroll
    for (int i = 0; i < TR; ++i) a_at[i][j] = (uint32_t)((group * TR + i) * 128 + ((j ^ ((group * TR + i) & 7)) << 4));
  }
  float acc[TR];
#pragma unroll
  for (int i = 0; i < TR; ++i) acc[i] = 0.f;
  constexpr int KS = TR <= 2 ? 4 : (TR <= 4 ? 2 : 1), BLOCKS = C::KC / 4 / KS;
  for (int c = 0; c < chunks; ++c) {
    const bool ok = mbar_wait(&full[c % ST], (c / ST) & 1, abort_flag);
    if (!__all_sync(0xffffffffu, ok)) {
      if (lane == 0) { *abort_flag = 1; atomicExch(status, ERR_SK_CONSUMER); }
      return;
    }
    const uint32_t wb = smem_u32(sm) + (c % ST) * C::STAGE, ab = wb + KB * C::W_BOX;
    float4 wv[2][KS], av[2][KS][TR];
    auto read = [&](int block) {
#pragma unroll
      for (int j = 0; j < KS; ++j) {
        const int piece = block * KS + j;
        wv[block & 1][j] = read_shared4(wb + piece / 8 * C::W_BOX + w_at[piece % 8]);
#pragma unroll
        for (int i = 0; i < TR; ++i) av[block & 1][j][i] = read_shared4(ab + piece / 8 * C::A_STEP + a_at[i][piece % 8]);
      }
    };
    read(0);
#pragma unroll
    for (int block = 0; block < BLOCKS; ++block) {
      if (block + 1 < BLOCKS) read(block + 1);
#pragma unroll
      for (int j = 0; j < KS; ++j) {
        const float4 w4 = wv[block & 1][j];
        const float4* a4 = av[block & 1][j];
#pragma unroll
        for (int i = 0; i < TR; ++i) acc[i] = fmaf(a4[i].x, w4.x, acc[i]);
#pragma unroll
        for (int i = 0; i < TR; ++i) acc[i] = fmaf(a4[i].y, w4.y, acc[i]);
#pragma unroll
        for (int i = 0; i < TR; ++i) acc[i] = fmaf(a4[i].z, w4.z, acc[i]);
#pragma unroll
        for (int i = 0; i < TR; ++i) acc[i] = fmaf(a4[i].w, w4.w, acc[i]);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[c % ST]);
  }
  if (!computes || n0 + row >= n) return;
#pragma unroll
  for (int i = 0; i < TR; ++i) {
    const int gm = m0 + group * TR + i;
    if (gm >= m) continue;
    const size_t o = (size_t)gm * ldo + n0 + row;
    if (MODE == OUT_ACC) out[o] += acc[i];
    else out[o] = acc[i];
  }
}

// A float32 matrix [rows, k] with row stride ld, in boxes of `box` rows x 32 values.
static bool make_skinny_map(CUtensorMap* map, const float* ptr, int rows, int k, long long ld, int box) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t boxes[2] = {32u, (cuuint32_t)box};
  cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, boxes, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int R, int RW, int TR, int W, int KB, int ST>
int launch_skinny(const float* a, const float* w, float* out, int m, int n, int k, int lda, int ldo, int mode, int* status, cudaStream_t s) {
  using C = Skinny<R, RW, TR, W, KB, ST>;
  TLLM_RESERVE_SMEM("linear_skinny", C::SMEM, (linear_skinny_kernel<R, RW, TR, W, KB, ST, OUT_ACC>), (linear_skinny_kernel<R, RW, TR, W, KB, ST, OUT_F32>));
  CUtensorMap mw, ma;
  if (!make_skinny_map(&mw, w, n, k, k, C::ROWS) || !make_skinny_map(&ma, a, m, k, lda, R))
    TLLM_FAIL(TLLM_ERR_CUDA, "linear_skinny: cuTensorMapEncodeTiled failed");
  dim3 grid((n + C::ROWS - 1) / C::ROWS, (m + R - 1) / R);
  if (mode == OUT_ACC)
    TLLM_LAUNCH("linear_skinny", (linear_skinny_kernel<R, RW, TR, W, KB, ST, OUT_ACC>), grid, W * 32 + 32, C::SMEM, s, mw, ma, out, m, n, k, ldo, status);
  else
    TLLM_LAUNCH("linear_skinny", (linear_skinny_kernel<R, RW, TR, W, KB, ST, OUT_F32>), grid, W * 32 + 32, C::SMEM, s, mw, ma, out, m, n, k, ldo, status);
  return TLLM_OK;
}

// Which shape: few weight rows want small CTAs (more SMs at work), many want the weight rows' reads shared by more rows of A.
// A wave of the small CTAs is 4,736 weight rows at m = 5 to 8 (four per SM), of the large ones 14,208, and a large one takes
// about twice as long.  K = 2,048, us, small / large, weights not in the L2:
//   weight rows   2,048        4,096        5,120        8,192        10,240       16,384       32,000
//   m = 1         7.6 / 10.6   9.1 / 11.2   16 / 12      18 / 13      26 / 24      35 / 26      65 / 51
//   m = 8         13 / 21      14 / 24      25 / 26      29 / 27      41 / 28      56 / 54      99 / 83
//   m = 16        19 / 33      20 / 40      38 / 42      40 / 44      59 / 45      80 / 88      140 / 133
// So the line may lie anywhere from 4,736 to 9,472 for eight rows; one row would take the large shape from 4,736 on, and 16
// rows the small one up to 9,472.  (K = 5,632 gives the same picture.)  Two to four rows were measured in one shape only.
static int launch_skinny_rows(const float* a, const float* w, float* out, int m, int n, int k, int lda, int ldo, int mode, int* status, cudaStream_t s) {
  const bool many = n >= 8192;
  if (m <= 1) return many ? launch_skinny<1, 32, 1, 1, 2, 8>(a, w, out, m, n, k, lda, ldo, mode, status, s)
                          : launch_skinny<1, 16, 1, 1, 4, 8>(a, w, out, m, n, k, lda, ldo, mode, status, s);
  if (m <= 2) return launch_skinny<2, 16, 1, 2, 4, 5>(a, w, out, m, n, k, lda, ldo, mode, status, s);
  if (m <= 4) return launch_skinny<4, 8, 1, 2, 4, 6>(a, w, out, m, n, k, lda, ldo, mode, status, s);
  if (m <= 8) return many ? launch_skinny<8, 16, 4, 2, 2, 6>(a, w, out, m, n, k, lda, ldo, mode, status, s)
                          : launch_skinny<8, 8, 2, 1, 4, 6>(a, w, out, m, n, k, lda, ldo, mode, status, s);
  return many ? launch_skinny<16, 16, 8, 2, 2, 6>(a, w, out, m, n, k, lda, ldo, mode, status, s)
              : launch_skinny<16, 8, 4, 2, 4, 5>(a, w, out, m, n, k, lda, ldo, mode, status, s);
}

template <typename T>
int launch(const void* a, const void* w, void* out, int m, int n, int k, int lda, int ldo, int mode, cudaStream_t s) {
  dim3 grid((n + BN - 1) / BN, (m + BM - 1) / BM);
  if (mode == OUT_SAME)
    TLLM_LAUNCH("linear_generic", (linear_generic_kernel<T, OUT_SAME>), grid, THREADS, 0, s, (const T*)a, (const T*)w, out, m, n, k, lda, ldo);
  else if (mode == OUT_F32)
    TLLM_LAUNCH("linear_generic", (linear_generic_kernel<T, OUT_F32>), grid, THREADS, 0, s, (const T*)a, (const T*)w, out, m, n, k, lda, ldo);
  else if (mode == OUT_ACC)
    TLLM_LAUNCH("linear_generic", (linear_generic_kernel<T, OUT_ACC>), grid, THREADS, 0, s, (const T*)a, (const T*)w, out, m, n, k, lda, ldo);
  else
    TLLM_FAIL(TLLM_ERR_ARG, "linear: unknown output mode %d", mode);
  return TLLM_OK;
}

}  // namespace tllm

// skinny: 0 keeps the 64 x 64 tile kernel for every size (tests compare it with the two others, which must agree with it to the bit)
extern "C" int tllm_linear_generic(const void* a, const void* w, void* out, int m, int n, int k, int lda, int ldo,
                                   int dtype, int mode, int skinny, int* status, void* stream) {
  TLLM_REQUIRE(m > 0 && n > 0 && k > 0, "linear: empty product %d x %d x %d", m, n, k);
  TLLM_REQUIRE(lda >= k && ldo >= n, "linear: row strides %d, %d are shorter than the rows %d, %d", lda, ldo, k, n);
  TLLM_REQUIRE((m + tllm::BM - 1) / tllm::BM <= 65535, "linear: %d rows exceed the grid", m);
  if (dtype == TLLM_F32 && m <= 16 && skinny != 0 && status != nullptr && k % 4 == 0 && lda % 4 == 0 && ((uintptr_t)a % 16) == 0 && ((uintptr_t)w % 16) == 0 &&
      (mode == tllm::OUT_SAME || mode == tllm::OUT_F32 || mode == tllm::OUT_ACC)) {
    const float* af = (const float*)a;
    const float* wf = (const float*)w;
    float* of = (float*)out;
    cudaStream_t s = (cudaStream_t)stream;
    return tllm::launch_skinny_rows(af, wf, of, m, n, k, lda, ldo, mode, status, s);
  }
  if (dtype == TLLM_F32 && skinny != 0 && m > 16 && k % 4 == 0 && lda % 4 == 0 && ((uintptr_t)a % 16) == 0 && ((uintptr_t)w % 16) == 0 &&
      n <= 64 * 65535 && (mode == tllm::OUT_SAME || mode == tllm::OUT_F32 || mode == tllm::OUT_ACC))
    return tllm::launch_tiled((const float*)a, (const float*)w, (float*)out, m, n, k, lda, ldo, mode, (cudaStream_t)stream);
  if (dtype == TLLM_F32) return tllm::launch<float>(a, w, out, m, n, k, lda, ldo, mode, (cudaStream_t)stream);
  if (dtype == TLLM_BF16) return tllm::launch<__nv_bfloat16>(a, w, out, m, n, k, lda, ldo, mode, (cudaStream_t)stream);
  TLLM_FAIL(TLLM_ERR_ARG, "linear: unknown dtype code %d", dtype);
}
