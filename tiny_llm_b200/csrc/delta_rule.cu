// The gated delta rule: a matrix state per head that is decayed, corrected towards the current value and read out,
//   S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q            S: [key size, value size]
// with q and k unit vectors per head (q also times a constant), one decay g and one step size beta per head and
// token.  q, k and v come from short causal convolutions (one filter per channel) with SiLU behind them; the last
// taps - 1 inputs of every channel are part of the request's state, beside S.  Decays, step sizes, unit norms, the
// recurrence and the state are 32-bit; the projections are of the engine's dtype.
//
// Three variants share the kernels (`mode`):
//   0  the rule above with one decay per head and token;
//   1  a state-space recurrence without the correction, S <- g S + k (dt v)^T, o = S^T q, where the step size dt =
//      softplus(b + dt_bias) also sets the decay g = exp(-exp(A_log) dt), the convolutions have a bias, nothing is made
//      a unit vector, and the projection's channels come in the order [values | keys | queries];
//   2  the rule above with a decay per head, key channel and token, S <- diag(g) S, from a 32-bit input row of its own.
//
// delta_prepare: one warp per (token, head row).  The channels of the fused projection's row are
//   [kvh heads of queries | kvh heads of keys | heads of values | ...]; a row's channels are filtered over the
//   request's earlier tokens in this step and, ahead of them, the inputs kept in the state; SiLU; query and key rows
//   are divided by sqrt(sum(x^2) + unit_eps); the value rows' warps also leave the head's decay and step size:
//   g = exp(-exp(A_log) softplus(a + dt_bias)), beta = sigmoid(b).  All outputs float32.
// conv_state_update: the state's kept inputs after the step: the last taps - 1 of (kept inputs ++ the step's, plus their
//   bias where the projection has one).
// delta_rule_scan: a group of 8 lanes owns one value column of one (request, head): the column's state rows lie in
//   the lanes' registers (a lane holds R consecutive rows).  Per token one round of shuffles gives the column's
//   S^T k, S^T q and k . q from the state as it was; with those
//       u = beta (v - g S^T k),   o = g S^T q + u (k . q),   S <- g S + k u
//   which is the sequence above with the read-out written in terms of the old state.  Tokens are staged in shared
//   memory eight at a time by cp.async, the next eight in flight meanwhile.  The state is kept transposed
//   ([slot, head, value column, key row]) so that a group's rows are consecutive in memory.  What is done to a state
//   element is the same sequence of operations however the request was cut into steps: the same bits.
// delta_rule_stream: the same for key rows of whole 16-byte pieces.  A bounded wait that runs out leaves a code in the
//   device's status word.
#include "tc_common.cuh"

TLLM_DEFINE_LAST_ERROR

namespace tllm {

__device__ __forceinline__ float softplus_f(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float silu_exact(float x) { return x / (1.f + expf(-x)); }

struct PrepArgs {
  const void* proj;            // [T, ld]: channels first, then whatever else the projection carries
  int ld;
  const float* taps;           // [channels, n_taps]: the last column meets the current token
  int n_taps;
  const float* kept;           // [slots, n_taps - 1, channels]: inputs of the tokens before this step, oldest first
  const int* slots;
  const int* cu_q;
  const int* token_request;
  int heads, kv_heads, kd, vd;
  int beta_col, a_col;         // columns of the projection row that hold b and a (one per head each)
  const float* a_log;          // [heads]
  const float* dt_bias;        // [heads]
  float q_scale, unit_eps;
  float *q, *k, *v, *gb;       // [T, kv_heads * kd] x 2, [T, heads * vd], [T, heads, 2] = (decay, step size)
  int n_tokens;
  int q_c0, k_c0, v_c0;        // first channel of the queries, the keys and the values
  const float* conv_bias;      // [channels] or null
  int unit_norm;               // query and key heads are made unit vectors
  int mode;                    // see the top of the file
  const float* a_in;           // mode 2: [T, heads * kd] inputs of the decays (dt_bias has heads * kd values then)
  float* gk;                   // mode 2: [T, heads * kd] decays
};

template <typename T>
__global__ void __launch_bounds__(128) delta_prepare_kernel(PrepArgs a) {
  pdl_trigger();
  pdl_wait();
  const int units = 2 * a.kv_heads + a.heads;
  const long long task = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (task >= (long long)a.n_tokens * units) return;
  const int lane = threadIdx.x & 31;
  const int t = (int)(task / units), u = (int)(task % units);
  const int req = a.token_request[t];
  const int first = a.cu_q[req];
  const int channels = 2 * a.kv_heads * a.kd + a.heads * a.vd;
  const float* kept = a.kept + (size_t)a.slots[req] * (a.n_taps - 1) * channels;
  const T* proj = (const T*)a.proj;
  int c0, size;
  float* dst;
  const bool is_v = u >= 2 * a.kv_heads;
  if (!is_v) {
    const bool is_q = u < a.kv_heads;
    const int hh = is_q ? u : u - a.kv_heads;
    c0 = (is_q ? a.q_c0 : a.k_c0) + hh * a.kd; size = a.kd;
    dst = (is_q ? a.q : a.k) + (size_t)t * a.kv_heads * a.kd + (size_t)hh * a.kd;
  } else {
    const int h = u - 2 * a.kv_heads;
    c0 = a.v_c0 + h * a.vd; size = a.vd;
    dst = a.v + (size_t)t * a.heads * a.vd + (size_t)h * a.vd;
  }
  float ss = 0.f;
  for (int d = lane; d < size; d += 32) {
    const int c = c0 + d;
    float y = a.conv_bias ? a.conv_bias[c] : 0.f;
    for (int j = 0; j < a.n_taps; ++j) {
      const int n = t - first - (a.n_taps - 1) + j;   // index among the request's tokens of this step; < 0: kept ones
      const float x = n >= 0 ? to_f32(proj[(size_t)(first + n) * a.ld + c])
                             : kept[(size_t)(a.n_taps - 1 + n) * channels + c];
      y = fmaf(a.taps[(size_t)c * a.n_taps + j], x, y);
    }
    y = silu_exact(y);
    dst[d] = y;
    ss = fmaf(y, y, ss);
  }
  if (!is_v) {
    if (a.unit_norm) {
      ss = warp_sum(ss);
      const float f = (u < a.kv_heads ? a.q_scale : 1.f) / sqrtf(ss + a.unit_eps);
      __syncwarp();
      for (int d = lane; d < size; d += 32) dst[d] = __fmul_rn(dst[d], f);
    }
    return;
  }
  const int h = u - 2 * a.kv_heads;
  if (a.mode == 2) {
    const float rate = expf(a.a_log[h]);
    const size_t at = ((size_t)t * a.heads + h) * a.kd;
    for (int d = lane; d < a.kd; d += 32)
      a.gk[at + d] = expf(-rate * softplus_f(a.a_in[at + d] + a.dt_bias[h * a.kd + d]));
  }
  if (lane == 0) {
    const float zb = to_f32(proj[(size_t)t * a.ld + a.beta_col + h]);
    float* gb = a.gb + ((size_t)t * a.heads + h) * 2;
    if (a.mode == 1) {
      const float dt = softplus_f(zb + a.dt_bias[h]);
      gb[0] = expf(-expf(a.a_log[h]) * dt);
      gb[1] = dt;
    } else {
      gb[0] = a.mode == 2 ? 1.f : expf(-expf(a.a_log[h]) * softplus_f(to_f32(proj[(size_t)t * a.ld + a.a_col + h]) + a.dt_bias[h]));
      gb[1] = 1.f / (1.f + expf(-zb));
    }
  }
}

// One thread per (request, channel): kept[j] <- input at (the request's tokens after this step) - (n_taps - 1) + j.
// Ascending j reads only entries at or above the one it writes, so the update is done in place.
template <typename T>
__global__ void conv_state_update_kernel(const T* __restrict__ proj, int ld, float* __restrict__ kept_all,
                                         const int* __restrict__ slots, const int* __restrict__ cu_q, int n_taps,
                                         int channels, int n_requests, const float* __restrict__ bias) {
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int req = blockIdx.y;
  if (c >= channels || req >= n_requests) return;
  const int first = cu_q[req], n = cu_q[req + 1] - first;
  float* kept = kept_all + (size_t)slots[req] * (n_taps - 1) * channels;
  const float add = bias ? bias[c] : 0.f;
  for (int j = 0; j < n_taps - 1; ++j) {
    const int i = n - (n_taps - 1) + j;   // index among this step's tokens; < 0: an input kept before
    kept[(size_t)j * channels + c] = i >= 0 ? to_f32(proj[(size_t)(first + i) * ld + c]) + add : kept[(size_t)(j + n) * channels + c];
  }
}

constexpr int DR_LANES = 8;            // lanes that share a value column
constexpr int DR_COLS = 16;            // value columns per CTA of 128 threads
constexpr int DR_TOK = 8;              // tokens staged at once

struct ScanArgs {
  const float *q, *k, *v, *gb;   // as delta_prepare leaves them
  float* state;                  // [slots, heads, vd, kd]
  const int* slots;
  const int* cu_q;
  float* out;                    // [T, heads * vd]
  int heads, kv_heads, kd, vd;
  const float* gk;               // mode 2: [T, heads * kd] decays per key channel
};

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int R, int MODE>   // R: state rows per lane, a multiple of 4: R * DR_LANES >= key size; MODE: see the top of the file
__global__ void __launch_bounds__(128) delta_rule_scan_kernel(ScanArgs a) {
  // A lane owns R consecutive state rows of its column (rows sub * R ... sub * R + R - 1), so that its part of a key
  // or query is read from shared memory in 16-byte pieces; a lane's part lies R + 4 floats from the next lane's, which
  // spreads the eight lanes of a column over all banks.
  constexpr int CH = R + 4;
  constexpr int KP = CH * DR_LANES;
  // per stage: q and k of DR_TOK tokens (rows past the key size stay zero), their values of this CTA's columns,
  // decay and step size
  __shared__ __align__(16) float sq[2][DR_TOK][KP], sk[2][DR_TOK][KP];
  __shared__ float sv[2][DR_TOK][DR_COLS], sg[2][DR_TOK][2];
  // decays per key channel: staged like q and k, except for the largest keys, whose three arrays would not fit a CTA's
  // static shared memory; those read their decays from global memory (the L1 holds a token's row for the CTA's columns)
  constexpr bool STAGED_DECAY = MODE == 2 && R < 32;
  __shared__ __align__(16) float sd[STAGED_DECAY ? 2 : 1][STAGED_DECAY ? DR_TOK : 1][STAGED_DECAY ? KP : 4];
  pdl_trigger();
  const int tid = threadIdx.x;
  const int sub = tid & (DR_LANES - 1), cl = tid / DR_LANES;
  const int h = blockIdx.y, req = blockIdx.z;
  const int col = blockIdx.x * DR_COLS + cl;
  const bool col_ok = col < a.vd;
  const int kh = h / (a.heads / a.kv_heads);
  for (int i = tid; i < 2 * DR_TOK * KP; i += 128) { (&sq[0][0][0])[i] = 0.f; (&sk[0][0][0])[i] = 0.f; }
  for (int i = tid; i < 2 * DR_TOK * DR_COLS; i += 128) (&sv[0][0][0])[i] = 0.f;
  if (STAGED_DECAY) for (int i = tid; i < 2 * DR_TOK * KP; i += 128) (&sd[0][0][0])[i] = 0.f;
  pdl_wait();
  const int t0 = a.cu_q[req], t1 = a.cu_q[req + 1];
  float* st = a.state + (((size_t)a.slots[req] * a.heads + h) * a.vd + (col_ok ? col : 0)) * a.kd;
  float s[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = sub * R + i;
    s[i] = (col_ok && row < a.kd) ? st[row] : 0.f;
  }
  __syncthreads();   // the zeros are in place before any copy lands beside them
  const int qk_ld = a.kv_heads * a.kd, v_ld = a.heads * a.vd;
  // 16-byte copies when a key row is made of whole pieces that start on 16-byte boundaries
  const bool wide = (a.kd & 3) == 0 && ((((size_t)a.q) | ((size_t)a.k) | ((size_t)a.gk)) & 15) == 0;
  const int g_ld = a.heads * a.kd;
  auto stage = [&](int buf, int tb) {
    const int nt = min(DR_TOK, t1 - tb);
    if (wide) {
      const int per = a.kd >> 2;
      for (int i = tid; i < nt * per; i += 128) {
        const int tt = i / per, d = (i - tt * per) << 2;
        const int at = (d / R) * CH + d % R;
        const size_t src = (size_t)(tb + tt) * qk_ld + (size_t)kh * a.kd + d;
        cp_async16(&sq[buf][tt][at], a.q + src);
        cp_async16(&sk[buf][tt][at], a.k + src);
        if (STAGED_DECAY) cp_async16(&sd[buf][tt][at], a.gk + (size_t)(tb + tt) * g_ld + (size_t)h * a.kd + d);
      }
    } else {
      for (int i = tid; i < nt * a.kd; i += 128) {
        const int tt = i / a.kd, d = i - tt * a.kd;
        const int at = (d / R) * CH + d % R;
        const size_t src = (size_t)(tb + tt) * qk_ld + (size_t)kh * a.kd + d;
        cp_async4(&sq[buf][tt][at], a.q + src);
        cp_async4(&sk[buf][tt][at], a.k + src);
        if (STAGED_DECAY) cp_async4(&sd[buf][tt][at], a.gk + (size_t)(tb + tt) * g_ld + (size_t)h * a.kd + d);
      }
    }
    for (int i = tid; i < nt * DR_COLS; i += 128) {
      const int tt = i / DR_COLS, c = i % DR_COLS;
      if (blockIdx.x * DR_COLS + c < a.vd)
        cp_async4(&sv[buf][tt][c], a.v + (size_t)(tb + tt) * v_ld + (size_t)h * a.vd + blockIdx.x * DR_COLS + c);
    }
    for (int i = tid; i < nt * 2; i += 128)
      cp_async4(&sg[buf][i / 2][i % 2], a.gb + ((size_t)(tb + i / 2) * a.heads + h) * 2 + i % 2);
  };
  auto fetch = [&](int buf, int tt, float* kr, float* qr) {   // this lane's part of a staged token's key and query
#pragma unroll
    for (int i = 0; i < R; i += 4) {
      const float4 kv = *reinterpret_cast<const float4*>(&sk[buf][tt][sub * CH + i]);
      const float4 qv = *reinterpret_cast<const float4*>(&sq[buf][tt][sub * CH + i]);
      kr[i] = kv.x; kr[i + 1] = kv.y; kr[i + 2] = kv.z; kr[i + 3] = kv.w;
      qr[i] = qv.x; qr[i + 1] = qv.y; qr[i + 2] = qv.z; qr[i + 3] = qv.w;
    }
  };
  stage(0, t0);
  cp_commit();
  int buf = 0;
  for (int tb = t0; tb < t1; tb += DR_TOK, buf ^= 1) {
    if (tb + DR_TOK < t1) stage(buf ^ 1, tb + DR_TOK);
    cp_commit();
    cp_wait<1>();
    __syncthreads();
    const int nt = min(DR_TOK, t1 - tb);
    float kn[R], qn[R];
    fetch(buf, 0, kn, qn);
    auto token = [&](int tt, bool more) {
      float kr[R], qr[R];
#pragma unroll
      for (int i = 0; i < R; ++i) { kr[i] = kn[i]; qr[i] = qn[i]; }
      if (more) fetch(buf, tt + 1, kn, qn);   // the next token's parts are on their way during this token's sums
      if (MODE == 2 && !STAGED_DECAY) {
        const float* gsrc = a.gk + (size_t)(tb + tt) * g_ld + (size_t)h * a.kd + sub * R;
#pragma unroll
        for (int i = 0; i < R; ++i)
          if (sub * R + i < a.kd) s[i] = __fmul_rn(s[i], __ldg(gsrc + i));
      }
      if (STAGED_DECAY) {   // the rows decay first, each by its own factor; the sums below then see the decayed state
#pragma unroll
        for (int i = 0; i < R; i += 4) {
          const float4 dv = *reinterpret_cast<const float4*>(&sd[buf][tt][sub * CH + i]);
          s[i] = __fmul_rn(s[i], dv.x); s[i + 1] = __fmul_rn(s[i + 1], dv.y);
          s[i + 2] = __fmul_rn(s[i + 2], dv.z); s[i + 3] = __fmul_rn(s[i + 3], dv.w);
        }
      }
      // four partial sums each, rows i, i + 4, i + 8, ... in one of them: short chains of dependent operations
      float pa[4] = {0.f, 0.f, 0.f, 0.f}, pb[4] = {0.f, 0.f, 0.f, 0.f}, pc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (MODE != 1) pa[i & 3] = fmaf(s[i], kr[i], pa[i & 3]);
        pb[i & 3] = fmaf(s[i], qr[i], pb[i & 3]);
        pc[i & 3] = fmaf(kr[i], qr[i], pc[i & 3]);
      }
      float xa = (pa[0] + pa[1]) + (pa[2] + pa[3]);
      float xb = (pb[0] + pb[1]) + (pb[2] + pb[3]);
      float xc = (pc[0] + pc[1]) + (pc[2] + pc[3]);
#pragma unroll
      for (int o = DR_LANES / 2; o > 0; o >>= 1) {
        xa += __shfl_xor_sync(0xffffffffu, xa, o);
        xb += __shfl_xor_sync(0xffffffffu, xb, o);
        xc += __shfl_xor_sync(0xffffffffu, xc, o);
      }
      const float g = sg[buf][tt][0], beta = sg[buf][tt][1];   // mode 2: g = 1, the rows have decayed already
      const float u = MODE == 1 ? __fmul_rn(beta, sv[buf][tt][cl]) : __fmul_rn(beta, fmaf(-g, xa, sv[buf][tt][cl]));
      const float o = fmaf(u, xc, __fmul_rn(g, xb));
#pragma unroll
      for (int i = 0; i < R; ++i) s[i] = fmaf(kr[i], u, __fmul_rn(g, s[i]));
      if (sub == 0 && col_ok) a.out[(size_t)(tb + tt) * v_ld + (size_t)h * a.vd + col] = o;
    };
    if (nt == DR_TOK) {   // a whole stage: unrolled, so that loads of later tokens can move ahead of earlier sums
#pragma unroll
      for (int tt = 0; tt < DR_TOK; ++tt) token(tt, tt + 1 < DR_TOK);
    } else {
      for (int tt = 0; tt < nt; ++tt) token(tt, tt + 1 < nt);
    }
    __syncthreads();   // the stage is free for the copies after the next
  }
  cp_wait<0>();
  if (col_ok) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = sub * R + i;
      if (row < a.kd) st[row] = s[i];
    }
  }
}


// The same recurrence, to the bit, where a key row is whole 16-byte pieces.  What bounded the kernel above was not its chain
// per token (two rounds of products and three of shuffles, about 150 cycles) but what stood between the chains: the
// copies' address arithmetic in every thread, two block barriers per eight tokens, three sums shuffled where the chain
// needs one.  Here a producer warp fills a ring of stages of eight tokens (a 16-byte piece of a row per lane), state rows
// go in pairs through fma.rn.f32x2, the tokens' values, decays and step sizes wait in registers, a token per lane, for a
// shuffle, and what only the read-out needs is summed for eight tokens at once.  (Two columns per lane, which halve the
// reads of shared memory, were slower, 378 us against 335: the chain then carries twice the products.)
// us for 1,777 tokens of 128 x 128, this kernel / the one above: mode 0, 16 heads 278 / 391; mode 1, 32 heads 328 / 450;
// mode 2, 16 heads 332 / 447; keys of 200, mode 2, 200 tokens 36 / 196; 61 tokens 18 / 24.
__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 halves_of(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {   // each half rounds like fmaf
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
constexpr int DR_STAGES = 4;

template <int R, int MODE>
struct Stream {
  static constexpr int WARPS = DR_COLS * DR_LANES / 32;
  static constexpr int ARRAYS = MODE == 2 ? 3 : 2, CH = R + 4, ROW = CH * DR_LANES;   // a lane's part of a staged row, padded (see above); the row
  static constexpr int STAGE = ARRAYS * DR_TOK * ROW;
  static constexpr int SMEM = DR_STAGES * STAGE * 4 + 2 * DR_STAGES * 8 + 16;
};

// x[t] of the eight lanes of a group summed per t in the tree of shuffles 4, 2, 1 apart; lane `sub` gets the sum of x[sub].
__device__ __forceinline__ float sum_per_token(float (&x)[DR_TOK], int sub) {
  static_assert(DR_TOK == 8 && DR_LANES == 8, "a token per lane");
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    const bool upper = (sub & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float keep = upper ? x[o + i] : x[i], give = upper ? x[i] : x[o + i];
      x[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  return x[0];
}

template <int R, int MODE>   // R * DR_LANES >= key size
__global__ void __launch_bounds__(Stream<R, MODE>::WARPS * 32 + 32) delta_rule_stream_kernel(ScanArgs a, int* __restrict__ status) {
  using C = Stream<R, MODE>;
  extern __shared__ __align__(16) float dr_smem[];     // [stage][keys, queries, decays][token][ROW]
  uint64_t* full = reinterpret_cast<uint64_t*>(dr_smem + DR_STAGES * C::STAGE);
  uint64_t* empty = full + DR_STAGES;
  volatile uint32_t* abort_flag = reinterpret_cast<uint32_t*>(empty + DR_STAGES);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.y, req = blockIdx.z, kh = h / (a.heads / a.kv_heads);
  if (tid == 0) {
    for (int s = 0; s < DR_STAGES; ++s) { mbar_init(&full[s], 32); mbar_init(&empty[s], C::WARPS); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (a.kd < R * DR_LANES)      // rows past the key size stay zero
    for (int i = tid; i < DR_STAGES * C::STAGE; i += C::WARPS * 32 + 32) dr_smem[i] = 0.f;
  __syncthreads();
  pdl_trigger();
  pdl_wait();
  const int t0 = a.cu_q[req], t1 = a.cu_q[req + 1], stages = (t1 - t0 + DR_TOK - 1) / DR_TOK;

  if (warp == C::WARPS) {
    // ---------------- producer: a lane copies the same pieces of every row
    const size_t qk_ld = (size_t)a.kv_heads * a.kd, g_ld = (size_t)a.heads * a.kd;
    for (int i = 0; i < stages; ++i) {
      const int s = i % DR_STAGES, tb = t0 + i * DR_TOK, nt = min(DR_TOK, t1 - tb);
      const bool ok = i < DR_STAGES || mbar_wait(&empty[s], ((i / DR_STAGES) & 1) ^ 1, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) { *abort_flag = 1; atomicExch(status, ERR_DR_PRODUCER); }
        break;
      }
      float* stage = dr_smem + s * C::STAGE;
#pragma unroll
      for (int d = lane * 4; d < R * DR_LANES; d += 128) {
        if (d >= a.kd) break;
        const int at = d / R * C::CH + d % R;
        const size_t qk = (size_t)tb * qk_ld + (size_t)kh * a.kd + d, gd = (size_t)tb * g_ld + (size_t)h * a.kd + d;
        for (int tt = 0; tt < nt; ++tt) {
          cp_async16(stage + tt * C::ROW + at, a.k + qk + tt * qk_ld);
          cp_async16(stage + (DR_TOK + tt) * C::ROW + at, a.q + qk + tt * qk_ld);
          if (MODE == 2) cp_async16(stage + (2 * DR_TOK + tt) * C::ROW + at, a.gk + gd + tt * g_ld);
        }
      }
      // arrives for this lane when its copies so far have landed
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[s])) : "memory");
    }
    cp_wait<0>();
    return;
  }

  const int sub = tid & (DR_LANES - 1), col = blockIdx.x * DR_COLS + tid / DR_LANES;
  const bool col_ok = col < a.vd;
  auto piece = [&](int j) { return sub * R + j * 4; };       // first row of this lane's j-th piece
  float* st = a.state + (((size_t)a.slots[req] * a.heads + h) * a.vd + col) * a.kd;
  uint64_t s[R / 2];
#pragma unroll
  for (int j = 0; j < R / 4; ++j) {
    ulonglong2 x = make_ulonglong2(0ull, 0ull);
    if (col_ok && piece(j) < a.kd) x = *reinterpret_cast<const ulonglong2*>(st + piece(j));
    s[2 * j] = x.x;
    s[2 * j + 1] = x.y;
  }
  const int v_ld = a.heads * a.vd;
  // values, decay and step size of token `sub` of a stage, in registers a stage ahead
  float v_next;
  float2 gb_next;
  auto ahead = [&](int tb) {
    const int t = tb + sub;
    v_next = t < t1 && col_ok ? a.v[(size_t)t * v_ld + (size_t)h * a.vd + col] : 0.f;
    gb_next = t < t1 ? *reinterpret_cast<const float2*>(a.gb + ((size_t)t * a.heads + h) * 2) : make_float2(0.f, 0.f);
  };
  ahead(t0);
  for (int i = 0; i < stages; ++i) {
    const int tb = t0 + i * DR_TOK, nt = min(DR_TOK, t1 - tb);
    const float v_now = v_next;
    const float2 gb_now = gb_next;
    ahead(tb + DR_TOK);
    const bool ok = mbar_wait(&full[i % DR_STAGES], (i / DR_STAGES) & 1, abort_flag);
    if (!__all_sync(0xffffffffu, ok)) {
      if (lane == 0) { *abort_flag = 1; atomicExch(status, ERR_DR_CONSUMER); }
      return;
    }
    const float* stage = dr_smem + (i % DR_STAGES) * C::STAGE + sub * C::CH;
    auto fetch = [&](int array, int tt, uint64_t* to) {
#pragma unroll
      for (int j = 0; j < R / 4; ++j) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(stage + (array * DR_TOK + tt) * C::ROW + j * 4);
        to[2 * j] = x.x;
        to[2 * j + 1] = x.y;
      }
    };
    uint64_t kn[R / 2], qn[R / 2];
    fetch(0, 0, kn);
    fetch(1, 0, qn);
    auto token = [&](int tt, bool more, float (&xb)[DR_TOK], float (&xc)[DR_TOK], float& u_mine) {
      uint64_t kr[R / 2], qr[R / 2];
#pragma unroll
      for (int j = 0; j < R / 2; ++j) { kr[j] = kn[j]; qr[j] = qn[j]; }
      if (more) { fetch(0, tt + 1, kn); fetch(1, tt + 1, qn); }   // the next token's parts are on their way during this token's sums
      if (MODE == 2) {   // the rows decay first, each by its own factor; the sums below then see the decayed state
        uint64_t d[R / 2];
        fetch(2, tt, d);
#pragma unroll
        for (int j = 0; j < R / 2; ++j) s[j] = mul2(s[j], d[j]);
      }
      // four partial sums each: short chains of dependent operations
      uint64_t pa[2] = {0ull, 0ull}, pb[2] = {0ull, 0ull}, pc[2] = {0ull, 0ull};
#pragma unroll
      for (int j = 0; j < R / 2; ++j) {
        if (MODE != 1) pa[j & 1] = fma2(s[j], kr[j], pa[j & 1]);
        pb[j & 1] = fma2(s[j], qr[j], pb[j & 1]);
        pc[j & 1] = fma2(kr[j], qr[j], pc[j & 1]);
      }
      auto joined = [](const uint64_t* p) {
        const float2 x = halves_of(p[0]), y = halves_of(p[1]);
        return (x.x + x.y) + (y.x + y.y);
      };
      // what the state's next value needs is summed over the group at once, the read-out at the end of the stage
      xc[tt] = joined(pc);
      xb[tt] = joined(pb);
      float xa = MODE != 1 ? joined(pa) : 0.f;
      if (MODE != 1) {
#pragma unroll
        for (int o = DR_LANES / 2; o > 0; o >>= 1) xa += __shfl_xor_sync(0xffffffffu, xa, o);
      }
      const int from = (lane & ~(DR_LANES - 1)) | tt;
      const float g = __shfl_sync(0xffffffffu, gb_now.x, from);   // mode 2: g = 1, the rows have decayed already
      const float beta = MODE == 1 ? 0.f : __shfl_sync(0xffffffffu, gb_now.y, from);
      const uint64_t gg = pair_of(g, g);
      float u;
      if (MODE == 1) {
        u = __shfl_sync(0xffffffffu, u_mine, from);
      } else {
        u = __fmul_rn(beta, fmaf(-g, xa, __shfl_sync(0xffffffffu, v_now, from)));
        if (sub == tt) u_mine = u;
      }
      const uint64_t uu = pair_of(u, u);
#pragma unroll
      for (int j = 0; j < R / 2; ++j) s[j] = fma2(kr[j], uu, mul2(gg, s[j]));
    };
    float xb[DR_TOK], xc[DR_TOK], u_mine = MODE == 1 ? __fmul_rn(gb_now.y, v_now) : 0.f;   // u_mine: of token `sub`
    if (nt == DR_TOK) {   // a whole stage without branches, so that loads of later tokens can move ahead of earlier sums
#pragma unroll
      for (int tt = 0; tt < DR_TOK; ++tt) token(tt, tt + 1 < DR_TOK, xb, xc, u_mine);
    } else {
#pragma unroll
      for (int tt = 0; tt < DR_TOK; ++tt) {
        xb[tt] = xc[tt] = 0.f;
        if (tt < nt) token(tt, tt + 1 < nt, xb, xc, u_mine);
      }
    }
    const float kq = sum_per_token(xc, sub);
    const float o = fmaf(u_mine, kq, __fmul_rn(gb_now.x, sum_per_token(xb, sub)));
    if (sub < nt && col_ok) a.out[(size_t)(tb + sub) * v_ld + (size_t)h * a.vd + col] = o;
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[i % DR_STAGES]);
  }
#pragma unroll
  for (int j = 0; j < R / 4; ++j)
    if (col_ok && piece(j) < a.kd) *reinterpret_cast<ulonglong2*>(st + piece(j)) = make_ulonglong2(s[2 * j], s[2 * j + 1]);
}

template <int R, int MODE>
static int launch_stream(const ScanArgs& a, dim3 grid, int* status, cudaStream_t s) {
  using C = Stream<R, MODE>;
  auto kern = delta_rule_stream_kernel<R, MODE>;
  TLLM_RESERVE_SMEM("delta_rule_scan", C::SMEM, kern);
  TLLM_LAUNCH("delta_rule_scan", kern, grid, C::WARPS * 32 + 32, C::SMEM, s, a, status);
  return TLLM_OK;
}

// gated_group_norm: y = (o + D_h x) * silu(z), then y / sqrt(mean(y^2) + eps) * w over each of `parts` equal parts of a
// token's row (a part need not be a head), in 32-bit; one CTA per (token, part).  o, x float32 [T, width] (x and D
// may be absent), z rows of ldz values in the engine's dtype, w float32 [width], out [T, width] in the engine's dtype.
template <typename T>
__global__ void __launch_bounds__(128) gated_group_norm_kernel(const float* __restrict__ o, const float* __restrict__ x,
                                                               const float* __restrict__ skip, const T* __restrict__ z,
                                                               int ldz, const float* __restrict__ w, T* __restrict__ out,
                                                               int width, int parts, int vd, float eps) {
  __shared__ float scratch[33];
  pdl_trigger();
  pdl_wait();
  const long long t = blockIdx.x / parts;
  const int part = blockIdx.x % parts, size = width / parts, c0 = part * size;
  const float* orow = o + t * width;
  const float* xrow = x ? x + t * width : nullptr;
  const T* zrow = z + t * ldz;
  auto value = [&](int c) {
    float y = orow[c];
    if (xrow) y = fmaf(skip[c / vd], xrow[c], y);
    const float g = to_f32(zrow[c]);
    return __fmul_rn(y, g / (1.f + expf(-g)));
  };
  float ss = 0.f;
  for (int i = threadIdx.x; i < size; i += blockDim.x) {
    const float y = value(c0 + i);
    ss = fmaf(y, y, ss);
  }
  ss = block_sum(ss, scratch);
  const float r = 1.f / sqrtf(ss / (float)size + eps);
  for (int i = threadIdx.x; i < size; i += blockDim.x)
    out[t * width + c0 + i] = from_f32<T>(__fmul_rn(__fmul_rn(value(c0 + i), r), w[c0 + i]));
}

}  // namespace tllm

using namespace tllm;

extern "C" int tllm_gated_group_norm(const float* o, const float* x, const float* skip, const void* z, int ldz,
                                     const float* w, void* out, long long n_tokens, int width, int parts, int vd,
                                     float eps, int dtype, void* stream) {
  TLLM_REQUIRE(n_tokens > 0 && width > 0 && parts > 0 && width % parts == 0 && vd > 0 && (x == nullptr) == (skip == nullptr),
               "gated_group_norm: %lld tokens, width %d in %d parts, heads of %d", n_tokens, width, parts, vd);
  const long long blocks = n_tokens * parts;
  TLLM_REQUIRE(blocks <= 2147483647LL, "gated_group_norm: %lld parts exceed the grid", blocks);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == TLLM_F32)
    TLLM_LAUNCH("gated_group_norm", gated_group_norm_kernel<float>, (unsigned)blocks, 128, 0, s, o, x, skip, (const float*)z, ldz, w, (float*)out, width, parts, vd, eps);
  else if (dtype == TLLM_BF16)
    TLLM_LAUNCH("gated_group_norm", gated_group_norm_kernel<__nv_bfloat16>, (unsigned)blocks, 128, 0, s, o, x, skip, (const __nv_bfloat16*)z, ldz, w, (__nv_bfloat16*)out, width, parts, vd, eps);
  else TLLM_FAIL(TLLM_ERR_ARG, "gated_group_norm: unknown dtype code %d", dtype);
  return TLLM_OK;
}

extern "C" int tllm_delta_prepare(const void* proj, int ld, const float* taps, int n_taps, const float* kept,
                                  const int* slots, const int* cu_q, const int* token_request, int heads, int kv_heads,
                                  int kd, int vd, int beta_col, int a_col, const float* a_log, const float* dt_bias,
                                  float q_scale, float unit_eps, float* q, float* k, float* v, float* gb, int n_tokens,
                                  int q_c0, int k_c0, int v_c0, const float* conv_bias, int unit_norm, int mode,
                                  const float* a_in, float* gk, int dtype, void* stream) {
  TLLM_REQUIRE(n_tokens > 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && kd > 0 && vd > 0 && n_taps >= 1,
               "delta_prepare: %d tokens, %d heads over %d query/key heads, sizes %d / %d, %d taps", n_tokens, heads, kv_heads, kd, vd, n_taps);
  PrepArgs a;
  a.proj = proj; a.ld = ld; a.taps = taps; a.n_taps = n_taps; a.kept = kept; a.slots = slots; a.cu_q = cu_q;
  a.token_request = token_request; a.heads = heads; a.kv_heads = kv_heads; a.kd = kd; a.vd = vd; a.beta_col = beta_col;
  a.a_col = a_col; a.a_log = a_log; a.dt_bias = dt_bias; a.q_scale = q_scale; a.unit_eps = unit_eps; a.q = q; a.k = k;
  a.v = v; a.gb = gb; a.n_tokens = n_tokens;
  TLLM_REQUIRE(mode >= 0 && mode <= 2 && (mode != 2 || (a_in && gk)), "delta_prepare: mode %d (0, 1 or 2; 2 needs the decays' inputs and outputs)", mode);
  a.q_c0 = q_c0; a.k_c0 = k_c0; a.v_c0 = v_c0; a.conv_bias = conv_bias; a.unit_norm = unit_norm; a.mode = mode; a.a_in = a_in; a.gk = gk;
  const long long tasks = (long long)n_tokens * (2 * kv_heads + heads);
  const long long blocks = (tasks + 3) / 4;
  TLLM_REQUIRE(blocks <= 2147483647LL, "delta_prepare: %lld rows exceed the grid", tasks);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == TLLM_F32) TLLM_LAUNCH("delta_prepare", delta_prepare_kernel<float>, (unsigned)blocks, 128, 0, s, a);
  else if (dtype == TLLM_BF16) TLLM_LAUNCH("delta_prepare", delta_prepare_kernel<__nv_bfloat16>, (unsigned)blocks, 128, 0, s, a);
  else TLLM_FAIL(TLLM_ERR_ARG, "delta_prepare: unknown dtype code %d", dtype);
  return TLLM_OK;
}

extern "C" int tllm_conv_state_update(const void* proj, int ld, float* kept, const int* slots, const int* cu_q, int n_taps,
                                      int channels, int n_requests, const float* bias, int dtype, void* stream) {
  TLLM_REQUIRE(n_requests > 0 && channels > 0 && n_taps >= 1 && n_requests <= 65535,
               "conv_state_update: %d requests, %d channels, %d taps", n_requests, channels, n_taps);
  if (n_taps == 1) return TLLM_OK;
  const dim3 grid((channels + 127) / 128, n_requests);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == TLLM_F32)
    TLLM_LAUNCH("conv_state_update", conv_state_update_kernel<float>, grid, 128, 0, s, (const float*)proj, ld, kept, slots, cu_q, n_taps, channels, n_requests, bias);
  else if (dtype == TLLM_BF16)
    TLLM_LAUNCH("conv_state_update", conv_state_update_kernel<__nv_bfloat16>, grid, 128, 0, s, (const __nv_bfloat16*)proj, ld, kept, slots, cu_q, n_taps, channels, n_requests, bias);
  else TLLM_FAIL(TLLM_ERR_ARG, "conv_state_update: unknown dtype code %d", dtype);
  return TLLM_OK;
}

extern "C" int tllm_delta_rule_scan(const float* q, const float* k, const float* v, const float* gb, float* state,
                                    const int* slots, const int* cu_q, float* out, int heads, int kv_heads, int kd, int vd,
                                    int n_requests, int n_tokens, int mode, const float* gk, int* status, void* stream) {
  TLLM_REQUIRE(n_requests > 0 && n_requests <= 65535 && heads > 0 && heads <= 65535 && kv_heads > 0 && heads % kv_heads == 0,
               "delta_rule_scan: %d requests, %d heads over %d query/key heads", n_requests, heads, kv_heads);
  TLLM_REQUIRE(kd >= 1 && kd <= 256 && vd >= 1, "delta_rule_scan: key size %d (at most 256), value size %d", kd, vd);
  ScanArgs a;
  a.q = q; a.k = k; a.v = v; a.gb = gb; a.state = state; a.slots = slots; a.cu_q = cu_q; a.out = out; a.heads = heads;
  a.kv_heads = kv_heads; a.kd = kd; a.vd = vd; a.gk = gk;
  TLLM_REQUIRE(mode >= 0 && mode <= 2 && (mode == 2) == (gk != nullptr), "delta_rule_scan: mode %d (0, 1 or 2; decays per key channel with 2 only)", mode);
  const dim3 grid((vd + DR_COLS - 1) / DR_COLS, heads, n_requests);
  cudaStream_t s = (cudaStream_t)stream;
  // The streamed kernel: key rows, decays and state columns of whole 16-byte pieces, and sizes where it is the faster one.
  // With key rows of less than 64 its fifth warp and its ring cost more than they save (us, streamed / general, values of 64,
  // keys of 36: 64 requests of one token, 32 heads, 38 / 22, of eight 56 / 43; 500 tokens 82 / 71; 32: 19 / 18, 39 / 37,
  // 76 / 67), except for the state-space form over portions, whose chain it shortens most (16: 500 tokens 47 / 55, 61 tokens
  // 7.4 / 8.7; eight requests of 16 12 / 10).  64: the streamed one (mode 1, 500 tokens 46 / 55; mode 2, 61 tokens 11.5 /
  // 12.8; decoded tokens 18 / 19), but for tokens of the delta rule where CTAs share SMs: 500 tokens 69 / 72 with 16 heads,
  // 82 / 72 with 32; eight requests of eight 4.3 / 4.9 with 8 heads, 6.4 / 5.9 with 16.  Above 64 it takes 0.2 to 0.9 of the
  // time (68 or 132 with 64 requests of one token and 32 heads 1.08).
  const bool decodes = n_tokens <= n_requests, portions = n_tokens >= 32LL * n_requests;
  const long long ctas = (long long)grid.x * heads * n_requests;
  const bool streamed = kd > 64 || (kd == 64 && (mode != 0 || decodes || ctas <= (portions ? 74 : 296))) || (mode == 1 && portions);
  if (streamed && (kd & 3) == 0 && status != nullptr && (((size_t)q | (size_t)k | (size_t)gk | (size_t)state) & 15) == 0 && ((size_t)gb & 7) == 0) {
#define TLLM_STREAM(R)                                                            \
  do {                                                                            \
    if (mode == 0) return launch_stream<R, 0>(a, grid, status, s);                \
    if (mode == 1) return launch_stream<R, 1>(a, grid, status, s);                \
    return launch_stream<R, 2>(a, grid, status, s);                               \
  } while (0)
    if (kd <= 32) return launch_stream<4, 1>(a, grid, status, s);   // (see above: mode 1 alone)
    if (kd <= 64) TLLM_STREAM(8);
    if (kd <= 128) TLLM_STREAM(16);
    TLLM_STREAM(32);
#undef TLLM_STREAM
  }
#define TLLM_SCAN(R)                                                                                         \
  do {                                                                                                       \
    if (mode == 0) TLLM_LAUNCH("delta_rule_scan", (delta_rule_scan_kernel<R, 0>), grid, 128, 0, s, a);       \
    else if (mode == 1) TLLM_LAUNCH("delta_rule_scan", (delta_rule_scan_kernel<R, 1>), grid, 128, 0, s, a);  \
    else TLLM_LAUNCH("delta_rule_scan", (delta_rule_scan_kernel<R, 2>), grid, 128, 0, s, a);                 \
  } while (0)
  if (kd <= 32) TLLM_SCAN(4);
  else if (kd <= 64) TLLM_SCAN(8);
  else if (kd <= 128) TLLM_SCAN(16);
  else TLLM_SCAN(32);
#undef TLLM_SCAN
  return TLLM_OK;
}
