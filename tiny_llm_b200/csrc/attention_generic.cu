// Attention of the step's queries over the paged cache on the CUDA cores, any key size up to 1,024 and any value
// size up to 512 (the two may differ; above 256 every (token, head) pair takes eight warps; key rows whose bytes are a multiple of 16 are read with 16-byte loads), any number of heads and groups, any
// page size.  It is the attention of the true 32-bit path and the fallback of the bfloat16 path.
//
// Heads.  A query head has `maps` score maps, each an attention of its own over the same values: the
// query rows of a token are laid out [head][map][kd], the key rows [key/value head][map][kd], the
// value rows [key/value head][vd]; map m of query head h reads key row (h / group) * maps + m and
// value row h / group, and the output rows are [head][map][vd].  maps = 1 is ordinary grouped-query
// attention.  The output is of the cache's type or float32 (for a caller that combines the maps).
//
// The keys a query at position p sees are j in [lo, p] with lo = max(0, p - window + 1) when there is a
// window and lo >= (p / chunk) * chunk when keys are visible inside a chunk of positions only (chunks
// are counted from position 0 of the sequence), and, with a window, also the sequence's first `keep` positions.  A score
// may get a learned bias by head and distance, rel[h][min(p - j, length - 1)] (added behind the scale).  They are walked in
// tiles of 32 that start at multiples of 32 of the absolute position.  Tile number i (= j / 32) belongs
// to lane i mod 8 of eight running softmaxes (m, l, o) in 32-bit, each of which takes its tiles in
// ascending order; at the end the eight are merged in the order 0..7.  So the order of every sum is a
// function of p alone: the result does not depend on how the request's tokens were cut into steps, on
// the rest of the batch or on the page ids.  Launches of the same arithmetic: float32 rows of up to 128 values that share
// their keys run several to a CTA (paged_attention_rows_kernel, below); else with many (token,
// head) pairs one warp carries all eight softmaxes of a pair (prompts); with few, eight warps carry
// one each and merge through shared memory (decoded tokens over a long context, where one warp per
// pair would leave most of the GPU idle and walk thousands of keys as one chain of memory latencies).
// Every step of both is written with explicit fmaf / __fmul_rn, so that the two compile to the same
// operations and give the same bits.
// Reference counterpart: tiny_llm/ops/cuda/flash_attention.cu:338-442 (64-key tiles,
// one lane per key, P.V by shuffles), whose mask compares a chunk-local query index with the
// absolute key index (:63-66, :402-405).
#include <math_constants.h>

#include "attention_route.h"
#include "common.cuh"

TLLM_DEFINE_LAST_ERROR

namespace tllm {

constexpr int WARPS = 4;
constexpr int MAX_HD = 256;            // sizes of all three launches
constexpr int MAX_KD = 1024, MAX_VD = 512;   // sizes of the launch with eight warps per pair

// Where the rows of the cache lie and which keys are visible; `nq` and `nk` count (head, map) rows.
struct Geometry {
  int nq, nk, maps, kd, vd, page_size, window, chunk;
  int keep;                 // keys j < keep are visible to every later token, whatever the window
  const float* rel;         // [query heads, rel_len]: what is added to a score at distance p - j (the last value beyond), or null
  int rel_len;
  int kvec;   // key rows are read with 16-byte loads (their size and strides allow it); else value by value, same order
  long long k_page_stride, k_head_stride, v_page_stride, v_head_stride;
};
__device__ __forceinline__ int lowest_key(const Geometry& g, int p) {
  int lo = g.window > 0 ? max(0, p - g.window + 1) : 0;
  if (g.chunk > 0) lo = max(lo, (p / g.chunk) * g.chunk);
  return lo;
}

template <typename T> struct Vec;            // 16-byte vectors of the cache rows
template <> struct Vec<float> { static constexpr int N = 4; };
template <> struct Vec<__nv_bfloat16> { static constexpr int N = 8; };

__device__ __forceinline__ void load16(const float* p, float* dst) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  dst[0] = v.x; dst[1] = v.y; dst[2] = v.z; dst[3] = v.w;
}
__device__ __forceinline__ void load16(const __nv_bfloat16* p, float* dst) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    dst[2 * i] = f.x; dst[2 * i + 1] = f.y;
  }
}

__device__ __forceinline__ float biased(const Geometry& g, float s, int head, int distance) {
  return g.rel == nullptr ? s : __fadd_rn(s, g.rel[(size_t)head * g.rel_len + min(distance, g.rel_len - 1)]);
}
// The tile after the one at j0 of the same way: tiles that lie wholly between the kept keys and the window are passed over.
__device__ __forceinline__ int next_tile(const Geometry& g, int j0, int step, int first_in_window) {
  const int n = j0 + step;
  return n >= g.keep ? max(n, first_in_window) : n;
}
// The same for the launches that walk whole groups of tiles together.
__device__ __forceinline__ bool tile_seen(const Geometry& g, int j0, int lo, int p) {
  return j0 <= p && (j0 + 31 >= lo || j0 < g.keep);
}

constexpr int WAYS = 8;   // running softmaxes per (token, head); a constant of the arithmetic, not a tuning knob

template <int OD>   // OD * 32 >= head size: the output values of a lane
struct Softmax {
  float m, l;
  float o[OD];
};

// One tile of 32 keys starting at j0 into the running softmax `st` (all lanes of the warp).
template <typename T, int OD>
__device__ __forceinline__ void attend_tile(Softmax<OD>& st, int j0, int lo, int p, const float* q_row, const T* kcache,
                                            const T* vcache, const int* table, int max_blocks, int kh, int vh,
                                            int head, const Geometry& g, int lane) {
  const int hd = g.kd, vd = g.vd, page_size = g.page_size;
  const int j = j0 + lane;
  bool valid = (j >= lo || j < g.keep) && j <= p && j / page_size < max_blocks;
  const int page = valid ? table[j / page_size] : -1;
  valid = valid && page >= 0;   // a table entry that names no page is never followed
  long long row_off = 0;
  float s = -CUDART_INF_F;
  if (valid) {
    row_off = (long long)page * g.v_page_stride + (long long)vh * g.v_head_stride + (long long)(j % page_size) * vd;
    const T* krow = kcache + (long long)page * g.k_page_stride + (long long)kh * g.k_head_stride + (long long)(j % page_size) * hd;
    float acc = 0.f;
    if (g.kvec) {
#pragma unroll 4
      for (int d = 0; d < hd; d += Vec<T>::N) {
        float kv[Vec<T>::N];
        load16(krow + d, kv);
#pragma unroll
        for (int e = 0; e < Vec<T>::N; ++e) acc = fmaf(q_row[d + e], kv[e], acc);
      }
    } else {
      for (int d = 0; d < hd; ++d) acc = fmaf(q_row[d], to_f32(krow[d]), acc);
    }
    s = biased(g, acc, head, p - j);
  }
  const float m_new = fmaxf(st.m, warp_max(s));
  const float m_ref = m_new == -CUDART_INF_F ? 0.f : m_new;   // a tile without a visible key changes nothing
  const float pr = valid ? expf(s - m_ref) : 0.f;
  const float corr = expf(st.m - m_ref);           // 0 on the first tile (m = -inf)
  st.l = fmaf(st.l, corr, warp_sum(pr));
  st.m = m_new;
#pragma unroll
  for (int i = 0; i < OD; ++i) st.o[i] = __fmul_rn(st.o[i], corr);
  const int last = min(31, p - j0);
  const int first = j0 < g.keep ? 0 : max(0, lo - j0);
  for (int kk = first; kk <= last; ++kk) {
    const float pk = __shfl_sync(0xffffffffu, pr, kk);
    if (pk == 0.f) continue;   // uniform across the warp: nothing to add, and the row may name no page
    const long long off = __shfl_sync(0xffffffffu, row_off, kk);
    const T* vrow = vcache + off;
#pragma unroll
    for (int i = 0; i < OD; ++i) {
      const int d = lane + 32 * i;
      if (d < vd) st.o[i] = fmaf(pk, to_f32(vrow[d]), st.o[i]);
    }
  }
}

// The merge of the eight softmaxes, way 0 first: `m`, `l`, `o` of way w are read through the three functions.
template <int OD, typename FM, typename FL, typename FO>
__device__ __forceinline__ void merge_ways(FM way_m, FL way_l, FO way_o, float* o_out, float& l_out, float& m_out) {
  float mx = -CUDART_INF_F;
#pragma unroll
  for (int w = 0; w < WAYS; ++w) mx = fmaxf(mx, way_m(w));
  const float m_ref = mx == -CUDART_INF_F ? 0.f : mx;
  m_out = m_ref;
  l_out = 0.f;
#pragma unroll
  for (int i = 0; i < OD; ++i) o_out[i] = 0.f;
#pragma unroll
  for (int w = 0; w < WAYS; ++w) {
    const float f = expf(way_m(w) - m_ref);   // 0 for a way that saw no key
    l_out = fmaf(way_l(w), f, l_out);
#pragma unroll
    for (int i = 0; i < OD; ++i) o_out[i] = fmaf(way_o(w, i), f, o_out[i]);
  }
}

// What the merged sums are multiplied by: 1 / l, or, with a sink (a learned score per head that joins the softmax's
// denominator and has no value), 1 / (l + exp(sink - m)) with both terms taken against the larger of m and the sink.
__device__ __forceinline__ float inverse_sum(float l, float m, const float* sink, int head) {
  if (sink == nullptr) return 1.f / l;
  const float sk = sink[head];
  const float top = fmaxf(m, sk);
  const float f = expf(m - top);
  return f / fmaf(l, f, expf(sk - top));
}

// The same tile for up to GH query heads that share the key/value head: every key row and value row is fetched once
// for all of them.  Head by head the operations are those of attend_tile, in the same order.
constexpr int GH = 4;

template <typename T, int OD>
__device__ __forceinline__ void attend_tile_grouped(Softmax<OD> (&st)[GH], int nh, int j0, int lo, int p,
                                                    const float (*q_rows)[OD * 32], const T* kcache, const T* vcache,
                                                    const int* table, int max_blocks, int kh, int vh, int head0,
                                                    const Geometry& g, int lane) {
  const int hd = g.kd, vd = g.vd, page_size = g.page_size;
  const int j = j0 + lane;
  bool valid = (j >= lo || j < g.keep) && j <= p && j / page_size < max_blocks;
  const int page = valid ? table[j / page_size] : -1;
  valid = valid && page >= 0;
  long long row_off = 0;
  float s[GH];
#pragma unroll
  for (int i = 0; i < GH; ++i) s[i] = -CUDART_INF_F;
  if (valid) {
    row_off = (long long)page * g.v_page_stride + (long long)vh * g.v_head_stride + (long long)(j % page_size) * vd;
    const T* krow = kcache + (long long)page * g.k_page_stride + (long long)kh * g.k_head_stride + (long long)(j % page_size) * hd;
    float acc[GH];
#pragma unroll
    for (int i = 0; i < GH; ++i) acc[i] = 0.f;
    if (g.kvec) {
#pragma unroll 2
      for (int d = 0; d < hd; d += Vec<T>::N) {
        float kv[Vec<T>::N];
        load16(krow + d, kv);
#pragma unroll
        for (int i = 0; i < GH; ++i)
#pragma unroll
          for (int e = 0; e < Vec<T>::N; ++e) acc[i] = fmaf(q_rows[i][d + e], kv[e], acc[i]);
      }
    } else {
      for (int d = 0; d < hd; ++d) {
        const float kvd = to_f32(krow[d]);
#pragma unroll
        for (int i = 0; i < GH; ++i) acc[i] = fmaf(q_rows[i][d], kvd, acc[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < GH; ++i) s[i] = i < nh ? biased(g, acc[i], head0 + i, p - j) : acc[i];
  }
  float pr[GH];
#pragma unroll
  for (int i = 0; i < GH; ++i) {
    pr[i] = 0.f;
    if (i < nh) {
      const float m_new = fmaxf(st[i].m, warp_max(s[i]));
      const float m_ref = m_new == -CUDART_INF_F ? 0.f : m_new;
      pr[i] = valid ? expf(s[i] - m_ref) : 0.f;
      const float corr = expf(st[i].m - m_ref);
      st[i].l = fmaf(st[i].l, corr, warp_sum(pr[i]));
      st[i].m = m_new;
#pragma unroll
      for (int x = 0; x < OD; ++x) st[i].o[x] = __fmul_rn(st[i].o[x], corr);
    }
  }
  const int last = min(31, p - j0);
  const int first = j0 < g.keep ? 0 : max(0, lo - j0);
  for (int kk = first; kk <= last; ++kk) {
    float pk[GH];
    bool any = false;
#pragma unroll
    for (int i = 0; i < GH; ++i) {
      pk[i] = __shfl_sync(0xffffffffu, pr[i], kk);
      any = any || pk[i] != 0.f;
    }
    if (!any) continue;   // uniform across the warp: nothing to add, and the row may name no page
    const long long off = __shfl_sync(0xffffffffu, row_off, kk);
    const T* vrow = vcache + off;
#pragma unroll
    for (int x = 0; x < OD; ++x) {
      const int d = lane + 32 * x;
      if (d < vd) {
        const float v = to_f32(vrow[d]);
#pragma unroll
        for (int i = 0; i < GH; ++i)
          if (pk[i] != 0.f) st[i].o[x] = fmaf(pk[i], v, st[i].o[x]);
      }
    }
  }
}

// Many (token, head) pairs (prompts): one warp per (token, key row, up to GH of the query rows that read it).  The eight
// softmaxes are walked one after the other (way w over its own tiles in ascending order, as everywhere), their results
// parked in shared memory and merged per head in the order 0..7: the arithmetic of every head is that of the other two
// launches, and the keys and values of a tile are fetched once for the heads of the group instead of once per head
// (with one warp per pair the kernel was bound by those fetches: 34 GB through L2 per layer of a 2,048-token prompt).
template <int OD> struct GroupedWarps { static constexpr int N = OD <= 2 ? 4 : (OD <= 4 ? 2 : 1); };

template <typename T, typename TO, int OD>
__global__ void __launch_bounds__(GroupedWarps<OD>::N * 32)
paged_attention_grouped_kernel(const T* __restrict__ q, int q_row_stride, const T* __restrict__ kcache,
                               const T* __restrict__ vcache, const int* __restrict__ block_table,
                               int max_blocks, const int* __restrict__ token_request,
                               const int* __restrict__ positions, TO* __restrict__ out, int n_tokens,
                               Geometry g, float scale, const float* __restrict__ sink) {
  constexpr int GW = GroupedWarps<OD>::N;
  __shared__ __align__(16) float q_s[GW][GH][OD * 32];
  __shared__ float way_s[GW][WAYS][GH][OD * 32 + 2];
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = g.nq, nk = g.nk, hd = g.kd, vd = g.vd, maps = g.maps;
  const int group = nq / nk, chunks = (group + GH - 1) / GH;
  const long long task = (long long)blockIdx.x * GW + warp;
  if (task >= (long long)n_tokens * nk * chunks) return;
  const int t = (int)(task / (nk * chunks)), rem = (int)(task % (nk * chunks));
  const int kh = rem / chunks, h0 = (rem % chunks) * GH, nh = min(GH, group - h0);
  const int kvh = kh / maps, map = kh % maps;   // query row of head h, map m: (h * maps + m)
  const int vh = kvh;
  const int req = token_request[t];
  const int p = positions[t];
  const int lo = lowest_key(g, p);
  const int* table = block_table + (size_t)req * max_blocks;
  for (int i = 0; i < nh; ++i) {
    const T* qrow = q + (size_t)t * q_row_stride + (size_t)((kvh * group + h0 + i) * maps + map) * hd;
    for (int d = lane; d < hd; d += 32) q_s[warp][i][d] = to_f32(qrow[d]) * scale;
  }
  for (int i = nh; i < GH; ++i)
    for (int d = lane; d < hd; d += 32) q_s[warp][i][d] = 0.f;
  __syncwarp();

  const int first_group = (lo / (32 * WAYS)) * (32 * WAYS), start = g.keep > 0 ? 0 : first_group;
  for (int w = 0; w < WAYS; ++w) {
    Softmax<OD> st[GH];
#pragma unroll
    for (int i = 0; i < GH; ++i) {
      st[i].m = -CUDART_INF_F; st[i].l = 0.f;
#pragma unroll
      for (int x = 0; x < OD; ++x) st[i].o[x] = 0.f;
    }
    for (int j0 = start + w * 32; j0 <= p; j0 = next_tile(g, j0, 32 * WAYS, first_group + w * 32))
      if (tile_seen(g, j0, lo, p))
        attend_tile_grouped<T, OD>(st, nh, j0, lo, p, q_s[warp], kcache, vcache, table, max_blocks, kh, vh, kvh * group + h0, g, lane);
#pragma unroll
    for (int i = 0; i < GH; ++i) {
      if (lane == 0) { way_s[warp][w][i][OD * 32] = st[i].m; way_s[warp][w][i][OD * 32 + 1] = st[i].l; }
#pragma unroll
      for (int x = 0; x < OD; ++x) way_s[warp][w][i][lane + 32 * x] = st[i].o[x];
    }
  }
  __syncwarp();
  for (int i = 0; i < nh; ++i) {
    float o[OD], l, mx;
    merge_ways<OD>([&](int w) { return way_s[warp][w][i][OD * 32]; }, [&](int w) { return way_s[warp][w][i][OD * 32 + 1]; },
                   [&](int w, int x) { return way_s[warp][w][i][lane + 32 * x]; }, o, l, mx);
    TO* orow = out + (size_t)t * nq * vd + (size_t)((kvh * group + h0 + i) * maps + map) * vd;
    const float inv = inverse_sum(l, mx, sink, kvh * group + h0 + i);
#pragma unroll
    for (int x = 0; x < OD; ++x) {
      const int d = lane + 32 * x;
      if (d < vd) orow[d] = from_f32<TO>(o[x] * inv);
    }
  }
}

// ---------------------------------------------------------------- float32: rows that share their keys in one CTA
// The same arithmetic for R rows at once, a row being a (token, query head of the key row's group) pair and consecutive
// rows consecutive pairs: a CTA of eight warps, warp w carrying way w of all rows.  What bounded the two launches above was
// fetching: a lane read its own key row 16 bytes at a time, and every value row was a trip to L2 that the next one waited
// for.  Here a tile's keys and values come to shared memory by cp.async (the next tile's while this one is worked on),
// once for all rows; a lane still is a key for the scores and a value column for the output, and the rows go in pairs
// through fma.rn.f32x2, whose halves round like fmaf.  The sums over a tile's 32 keys keep the tree of warp_sum: partners
// exchange halves of the rows instead of whole rows, so 16 rows take 16 steps of shuffles instead of 80 and 4 rows 6
// instead of 20.  us per layer at the TinyLlama sizes, this kernel / the launches above: a prompt of 509 tokens 110 / 351,
// eight decoded tokens at context 700 18 / 42.  What bounds it: the latencies of the eight warps that an SM has (the tiles
// take 144 to 164 KB, so one CTA); at 509 tokens issue slots are 27 % used, the load/store pipe 20 %, shared memory 34 %,
// and a quarter of a warp's time is the merge, where ways with fewer tiles wait.
__device__ __forceinline__ uint64_t pack_pair(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack_pair(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// v[r] of all 32 lanes reduced per row r in the tree of the butterflies warp_sum / warp_max (partners 16, 8, 4, 2, 1 apart);
// lane l gets the result of row l * R / 32.
template <int R, typename Op>
__device__ __forceinline__ float reduce_rows(const float (&in)[R], Op op, int lane) {
  float v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = in[r];
  int rows = R;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (rows > 1) {
      rows /= 2;
      const bool upper = (lane & o) != 0;
#pragma unroll
      for (int r = 0; r < R / 2; ++r)
        if (r < rows) {
          const float keep = upper ? v[rows + r] : v[r], give = upper ? v[r] : v[rows + r];
          v[r] = op(keep, __shfl_xor_sync(0xffffffffu, give, o));
        }
    } else {
      v[0] = op(v[0], __shfl_xor_sync(0xffffffffu, v[0], o));
    }
  }
  return v[0];
}

template <int OD, int R>
struct RowsSmem {
  // Keys and values of a tile in buffers of their own, or values over the keys that have been multiplied.  Sixteen rows of up
  // to 64 values: with one buffer two CTAs share an SM (92 KB of shared memory, 128 registers), and one computes while the
  // other waits; with two buffers one CTA had an SM for itself (32 heads over 4 of 64, us: 131 tokens 24.1 -> 16.6, 509
  // 108.9 -> 76.1, 2,048 1,007 -> 698, 300 beside eight decoded ones 107.7 -> 90.9).
  static constexpr bool TWO = OD <= 2 && R < 16;
  static constexpr int K_LD = OD * 32 + 4, V_LD = OD * 32, P_LD = R + 4;   // pitches that keep 16-byte accesses apart
  static constexpr int K_FLOATS = 32 * K_LD, V_FLOATS = TWO ? 32 * V_LD : 0, P_FLOATS = 32 * P_LD;
  static constexpr int WARP_FLOATS = K_FLOATS + V_FLOATS + P_FLOATS;
  static constexpr int Q_FLOATS = OD * 32 * R;
  static constexpr int MERGE_LD = OD * 32 + 2;
  static constexpr int BYTES = (WAYS * WARP_FLOATS + Q_FLOATS) * 4;
  static_assert(WAYS * R * MERGE_LD <= WAYS * WARP_FLOATS, "the ways' results are parked over the tiles");
};

template <int OD, int R>   // R = 4 or 16 rows
__global__ void __launch_bounds__(WAYS * 32)
paged_attention_rows_kernel(const float* __restrict__ q, int q_row_stride, const float* __restrict__ kcache,
                            const float* __restrict__ vcache, const int* __restrict__ block_table, int max_blocks,
                            const int* __restrict__ token_request, const int* __restrict__ positions,
                            float* __restrict__ out, int n_tokens, Geometry g, float scale, const float* __restrict__ sink) {
  using S = RowsSmem<OD, R>;
  extern __shared__ __align__(16) float rows_smem[];
  __shared__ int pos_s[R], lo_s[R], tok_s[R], head_s[R];   // token -1: no such row
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* q_s = rows_smem;                                   // [key value][row]
  float* k_s = rows_smem + S::Q_FLOATS + warp * S::WARP_FLOATS;   // [key][K_LD]
  float* v_s = S::TWO ? k_s + S::K_FLOATS : k_s;            // [key][V_LD]
  float* p_s = k_s + S::K_FLOATS + S::V_FLOATS;             // [key][P_LD]
  pdl_trigger();
  pdl_wait();
  const int kd = g.kd, vd = g.vd, maps = g.maps, page_size = g.page_size;
  const int group = g.nq / g.nk, kh = blockIdx.x % g.nk, vh = kh / maps, map = kh % maps;
  // a request's later tokens see more keys: the step's last rows start first (with decoded tokens ahead of a prompt, as the
  // scheduler lays a step out, those start last)
  const long long first = (long long)(gridDim.x / g.nk - 1 - blockIdx.x / g.nk) * R;
  const long long n_rows = (long long)n_tokens * group;
  const int t_first = (int)(first / group), t_last = (int)((min(first + R, n_rows) - 1) / group);
  if (threadIdx.x < R) {
    const long long row = first + threadIdx.x;
    const int t = (int)(row / group);
    const bool ok = row < n_rows;
    pos_s[threadIdx.x] = ok ? positions[t] : 0;
    lo_s[threadIdx.x] = ok ? lowest_key(g, positions[t]) : 0;
    tok_s[threadIdx.x] = ok ? t : -1;
    head_s[threadIdx.x] = vh * group + (int)(row % group);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < R * kd; i += WAYS * 32) {
    const int r = i / kd, d = i % kd;
    const bool ok = tok_s[r] >= 0;
    q_s[d * R + r] = ok ? q[(size_t)((first + r) / group) * q_row_stride + (size_t)(head_s[r] * maps + map) * kd + d] * scale : 0.f;
  }
  __syncthreads();

  uint64_t o[R / 2][OD];
#pragma unroll
  for (int r = 0; r < R / 2; ++r)
#pragma unroll
    for (int x = 0; x < OD; ++x) o[r][x] = 0ull;
  const int my_row = lane * R / 32;             // whose maximum and sum this lane keeps
  float m_run = -CUDART_INF_F, l_run = 0.f;

  // one request at a time (rows of a prompt have one; decoded tokens may have several): the others' rows see no key
  for (int t = t_first; t <= t_last;) {
    const int t_begin = t, req = token_request[t];
    while (t <= t_last && token_request[t] == req) ++t;
    const int t_end = t;
    int p_max = -1, p_min = 0x7fffffff, lo_min = 0x7fffffff, lo_max = 0;
    bool whole = true;                          // every row is of this request
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (tok_s[r] < t_begin || tok_s[r] >= t_end) { whole = false; continue; }
      p_max = max(p_max, pos_s[r]); p_min = min(p_min, pos_s[r]);
      lo_min = min(lo_min, lo_s[r]); lo_max = max(lo_max, lo_s[r]);
    }
    const int* table = block_table + (size_t)req * max_blocks;
    const int first_group = (lo_min / (32 * WAYS)) * (32 * WAYS) + warp * 32;
    auto seen_from = [&](int j0) {              // the first tile of this way from j0 on that some row sees
      while (j0 <= p_max && !tile_seen(g, j0, lo_min, p_max)) j0 = next_tile(g, j0, 32 * WAYS, first_group);
      return j0;
    };
    // this lane's key of the tile at j0: its page, or -1.  Every lane looks a page up (the last seen key's where it has no
    // key): with the lookup behind a branch the lanes with and without a key went through the scores and the softmax of the
    // tile before one after the other, 14 us on a request whose last tile of several is not whole (us per launch, eight
    // decoded tokens with 256 / 257 / 700 keys: 8.8 / 25.2 / 31.4, now 8.8 / 12.2 / 18.4)
    auto page_of = [&](int j0) {
      const int j = j0 + lane, block = min(j, p_max) / page_size, page = table[min(block, max_blocks - 1)];
      return (j <= p_max) & (block < max_blocks) ? page : -1;
    };
    // rows of the tile to shared memory, a row per OD * 8 lanes; keys without a page stay as they are and are not used
    auto fetch = [&](float* dst, int ld, const float* cache, long long page_stride, long long head_offset, int size, int j0, int page) {
      constexpr int LANES = OD * 8;
      const long long off = page < 0 ? -1 : (long long)page * page_stride + head_offset + (long long)((j0 + lane) % page_size) * size;
      const int c = (lane % LANES) * 4;
#pragma unroll 4
      for (int r0 = 0; r0 < 32; r0 += 32 / LANES) {
        const int r = r0 + lane / LANES;
        const long long at = __shfl_sync(0xffffffffu, off, r);
        if (at >= 0 && c < size) copy16_async(dst + r * ld + c, cache + at + c);
      }
      copies_commit();
    };
    const long long k_head = (long long)kh * g.k_head_stride, v_head = (long long)vh * g.v_head_stride;
    int j0 = seen_from(g.keep > 0 ? warp * 32 : first_group);
    int page = j0 <= p_max ? page_of(j0) : -1;
    if (j0 <= p_max) {
      fetch(k_s, S::K_LD, kcache, g.k_page_stride, k_head, kd, j0, page);
      if (S::TWO) fetch(v_s, S::V_LD, vcache, g.v_page_stride, v_head, vd, j0, page);
    }
    while (j0 <= p_max) {
      const int next = seen_from(next_tile(g, j0, 32 * WAYS, first_group));
      const int next_page = next <= p_max ? page_of(next) : -1;
      copies_wait<S::TWO ? 1 : 0>();
      __syncwarp();
      // ---- scores: this lane's key against all rows
      uint64_t acc[R / 2];
#pragma unroll
      for (int r = 0; r < R / 2; ++r) acc[r] = 0ull;
      const float* krow = k_s + lane * S::K_LD;
#pragma unroll 4
      for (int d = 0; d < kd; d += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(krow + d);
        const float kv[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint64_t kk = pack_pair(kv[e], kv[e]);
#pragma unroll
          for (int r = 0; r < R; r += 4) {
            const ulonglong2 q4 = *reinterpret_cast<const ulonglong2*>(q_s + (d + e) * R + r);
            acc[r / 2] = fma_pair(q4.x, kk, acc[r / 2]);
            acc[r / 2 + 1] = fma_pair(q4.y, kk, acc[r / 2 + 1]);
          }
        }
      }
      __syncwarp();
      if (S::TWO) {
        if (next <= p_max) fetch(k_s, S::K_LD, kcache, g.k_page_stride, k_head, kd, next, next_page);
        else copies_commit();
      } else {
        fetch(v_s, S::V_LD, vcache, g.v_page_stride, v_head, vd, j0, page);
      }
      // ---- softmax
      const int j = j0 + lane;
      const bool inside = whole && j0 + 31 <= p_min && j0 >= lo_max && __all_sync(0xffffffffu, page >= 0);
      float s[R], pr[R];
      uint32_t valid = 0xffffffffu;             // bit r: row r sees this lane's key
#pragma unroll
      for (int r = 0; r < R; r += 2) {
        const float2 two = unpack_pair(acc[r / 2]);
        s[r] = two.x;
        s[r + 1] = two.y;
      }
      if (!inside) {
        valid = 0;
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (tok_s[r] >= t_begin && tok_s[r] < t_end && page >= 0 && (j >= lo_s[r] || j < g.keep) && j <= pos_s[r]) valid |= 1u << r;
      }
      if (g.rel != nullptr) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (valid >> r & 1u) s[r] = biased(g, s[r], head_s[r], pos_s[r] - j);
      }
      if (!inside) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (!(valid >> r & 1u)) s[r] = -CUDART_INF_F;
      }
      const float m_new = fmaxf(m_run, reduce_rows<R>(s, [](float a, float b) { return fmaxf(a, b); }, lane));
      const float m_ref = m_new == -CUDART_INF_F ? 0.f : m_new;
      const float corr = expf(m_run - m_ref);
      m_run = m_new;
      bool none = true, every = true;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float ref = __shfl_sync(0xffffffffu, m_ref, r * 32 / R);
        pr[r] = valid >> r & 1u ? expf(s[r] - ref) : 0.f;
        none = none && pr[r] == 0.f;
        every = every && pr[r] != 0.f;
      }
      l_run = fmaf(l_run, corr, reduce_rows<R>(pr, [](float a, float b) { return a + b; }, lane));
#pragma unroll
      for (int r = 0; r < R; r += 4) *reinterpret_cast<float4*>(p_s + lane * S::P_LD + r) = make_float4(pr[r], pr[r + 1], pr[r + 2], pr[r + 3]);
      if (!__all_sync(0xffffffffu, corr == 1.f)) {
#pragma unroll
        for (int r = 0; r < R; r += 2) {
          const float c0 = __shfl_sync(0xffffffffu, corr, r * 32 / R), c1 = __shfl_sync(0xffffffffu, corr, (r + 1) * 32 / R);
#pragma unroll
          for (int x = 0; x < OD; ++x) {
            const float2 two = unpack_pair(o[r / 2][x]);
            o[r / 2][x] = pack_pair(__fmul_rn(two.x, c0), __fmul_rn(two.y, c1));
          }
        }
      }
      // keys that some row weighs, and keys that every row weighs (the others' products are left out row by row)
      const uint32_t some = ~__ballot_sync(0xffffffffu, none), all = __ballot_sync(0xffffffffu, every);
      copies_wait<S::TWO ? 1 : 0>();
      __syncwarp();
      // ---- output: this lane's value columns
      if (all == 0xffffffffu) {
#pragma unroll 4
        for (int kk = 0; kk < 32; ++kk) {
          ulonglong2 p4[R / 4];
#pragma unroll
          for (int r = 0; r < R / 4; ++r) p4[r] = *reinterpret_cast<const ulonglong2*>(p_s + kk * S::P_LD + 4 * r);
#pragma unroll
          for (int x = 0; x < OD; ++x) {
            const float v = v_s[kk * S::V_LD + lane + 32 * x];
            const uint64_t vv = pack_pair(v, v);
#pragma unroll
            for (int r = 0; r < R / 4; ++r) {
              o[2 * r][x] = fma_pair(p4[r].x, vv, o[2 * r][x]);
              o[2 * r + 1][x] = fma_pair(p4[r].y, vv, o[2 * r + 1][x]);
            }
          }
        }
      } else {
        for (uint32_t left = some; left != 0; left &= left - 1) {
          const int kk = __ffs(left) - 1;
#pragma unroll
          for (int x = 0; x < OD; ++x) {
            const float v = v_s[kk * S::V_LD + lane + 32 * x];
#pragma unroll
            for (int r = 0; r < R; r += 2) {
              const float2 p2 = *reinterpret_cast<const float2*>(p_s + kk * S::P_LD + r);
              float2 two = unpack_pair(o[r / 2][x]);
              if (p2.x != 0.f) two.x = fmaf(p2.x, v, two.x);
              if (p2.y != 0.f) two.y = fmaf(p2.y, v, two.y);
              o[r / 2][x] = pack_pair(two.x, two.y);
            }
          }
        }
      }
      __syncwarp();
      if (next <= p_max) {
        if (S::TWO) fetch(v_s, S::V_LD, vcache, g.v_page_stride, v_head, vd, next, next_page);
        else fetch(k_s, S::K_LD, kcache, g.k_page_stride, k_head, kd, next, next_page);
      }
      j0 = next;
      page = next_page;
    }
    copies_wait<0>();
    __syncwarp();
  }

  // ---- the ways of every row meet
  __syncthreads();
  float* merge_s = rows_smem + S::Q_FLOATS;     // [way][row][MERGE_LD]
  float* mine = merge_s + warp * R * S::MERGE_LD;
#pragma unroll
  for (int r = 0; r < R; r += 2)
#pragma unroll
    for (int x = 0; x < OD; ++x) {
      const float2 two = unpack_pair(o[r / 2][x]);
      mine[r * S::MERGE_LD + lane + 32 * x] = two.x;
      mine[(r + 1) * S::MERGE_LD + lane + 32 * x] = two.y;
    }
  if (lane % (32 / R) == 0) { mine[my_row * S::MERGE_LD + OD * 32] = m_run; mine[my_row * S::MERGE_LD + OD * 32 + 1] = l_run; }
  __syncthreads();
  for (int r = warp; r < R; r += WAYS) {
    if (tok_s[r] < 0) continue;
    float sums[OD], l, mx;
    auto way = [&](int w, int i) { return merge_s[(w * R + r) * S::MERGE_LD + i]; };
    merge_ways<OD>([&](int w) { return way(w, OD * 32); }, [&](int w) { return way(w, OD * 32 + 1); },
                   [&](int w, int x) { return way(w, lane + 32 * x); }, sums, l, mx);
    float* orow = out + (size_t)((first + r) / group) * g.nq * vd + (size_t)(head_s[r] * maps + map) * vd;
    const float inv = inverse_sum(l, mx, sink, head_s[r]);
#pragma unroll
    for (int x = 0; x < OD; ++x)
      if (lane + 32 * x < vd) orow[lane + 32 * x] = sums[x] * inv;
  }
}

template <int OD, int R>
static int launch_rows(const float* q, int q_row_stride, const float* kcache, const float* vcache, const int* block_table,
                       int max_blocks, const int* token_request, const int* positions, float* out, int n_tokens,
                       const Geometry& g, float scale, const float* sink, long long blocks, cudaStream_t s) {
  auto kern = paged_attention_rows_kernel<OD, R>;
  TLLM_RESERVE_SMEM("attention", (RowsSmem<OD, R>::BYTES), kern);
  TLLM_LAUNCH("paged_attention_rows", kern, (unsigned)blocks, WAYS * 32, (RowsSmem<OD, R>::BYTES), s, q, q_row_stride, kcache, vcache,
              block_table, max_blocks, token_request, positions, out, n_tokens, g, scale, sink);
  return TLLM_OK;
}

// SPLIT = false: WARPS (token, head) pairs per CTA, one warp each, eight softmaxes in its registers.
// SPLIT = true: one pair per CTA of eight warps, warp w carries softmax w.
template <typename T, typename TO, bool SPLIT, int OD>
__global__ void __launch_bounds__(SPLIT ? WAYS * 32 : WARPS * 32)
paged_attention_generic_kernel(const T* __restrict__ q, int q_row_stride, const T* __restrict__ kcache,
                               const T* __restrict__ vcache, const int* __restrict__ block_table,
                               int max_blocks, const int* __restrict__ token_request,
                               const int* __restrict__ positions, TO* __restrict__ out, int n_tokens,
                               Geometry g, float scale, const float* __restrict__ sink) {
  __shared__ __align__(16) float q_s[SPLIT ? 1 : WARPS][SPLIT ? MAX_KD : MAX_HD];
  __shared__ float merge_s[SPLIT ? WAYS : 1][SPLIT ? OD * 32 + 2 : 1];
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = g.nq, nk = g.nk, hd = g.kd, vd = g.vd, maps = g.maps;
  const long long task = SPLIT ? (long long)blockIdx.x : (long long)blockIdx.x * WARPS + warp;
  if (task >= (long long)n_tokens * nq) return;
  const int t = (int)(task / nq), h = (int)(task % nq);   // h: the (head, map) row of the queries
  const int vh = (h / maps) / (nq / nk);
  const int kh = vh * maps + h % maps;
  const int req = token_request[t];
  const int p = positions[t];
  const int lo = lowest_key(g, p);
  const int* table = block_table + (size_t)req * max_blocks;

  const T* qrow = q + (size_t)t * q_row_stride + (size_t)h * hd;
  float* q_row = q_s[SPLIT ? 0 : warp];
  if (SPLIT) {
    for (int d = threadIdx.x; d < hd; d += WAYS * 32) q_row[d] = to_f32(qrow[d]) * scale;
    __syncthreads();
  } else {
    for (int d = lane; d < hd; d += 32) q_row[d] = to_f32(qrow[d]) * scale;
    __syncwarp();
  }

  const int first_group = (lo / (32 * WAYS)) * (32 * WAYS);   // tile numbers are absolute: way = (j0 / 32) % WAYS
  const int start = g.keep > 0 ? 0 : first_group;
  float o[OD], l, mx;
  if (SPLIT) {
    Softmax<OD> st;
    st.m = -CUDART_INF_F; st.l = 0.f;
#pragma unroll
    for (int i = 0; i < OD; ++i) st.o[i] = 0.f;
    for (int j0 = start + warp * 32; j0 <= p; j0 = next_tile(g, j0, 32 * WAYS, first_group + warp * 32))
      if (tile_seen(g, j0, lo, p))
        attend_tile(st, j0, lo, p, q_row, kcache, vcache, table, max_blocks, kh, vh, h / maps, g, lane);
    if (lane == 0) { merge_s[warp][OD * 32] = st.m; merge_s[warp][OD * 32 + 1] = st.l; }
#pragma unroll
    for (int i = 0; i < OD; ++i)
      if (lane + 32 * i < vd) merge_s[warp][lane + 32 * i] = st.o[i];
    __syncthreads();
    if (warp != 0) return;
    merge_ways<OD>([&](int w) { return merge_s[w][OD * 32]; }, [&](int w) { return merge_s[w][OD * 32 + 1]; },
               [&](int w, int i) { return lane + 32 * i < vd ? merge_s[w][lane + 32 * i] : 0.f; }, o, l, mx);
  } else {
    Softmax<OD> st[WAYS];
#pragma unroll
    for (int w = 0; w < WAYS; ++w) {
      st[w].m = -CUDART_INF_F; st[w].l = 0.f;
#pragma unroll
      for (int i = 0; i < OD; ++i) st[w].o[i] = 0.f;
    }
    for (int g0 = start; g0 <= p; g0 = next_tile(g, g0, 32 * WAYS, first_group)) {
#pragma unroll
      for (int w = 0; w < WAYS; ++w) {
        const int j0 = g0 + w * 32;
        if (tile_seen(g, j0, lo, p))
          attend_tile(st[w], j0, lo, p, q_row, kcache, vcache, table, max_blocks, kh, vh, h / maps, g, lane);
      }
    }
    merge_ways<OD>([&](int w) { return st[w].m; }, [&](int w) { return st[w].l; }, [&](int w, int i) { return st[w].o[i]; }, o, l, mx);
  }
  TO* orow = out + (size_t)t * nq * vd + (size_t)h * vd;
  const float inv = inverse_sum(l, mx, sink, h / maps);
#pragma unroll
  for (int i = 0; i < OD; ++i) {
    const int d = lane + 32 * i;
    if (d < vd) orow[d] = from_f32<TO>(o[i] * inv);
  }
}

template <typename T, typename TO>
static int launch_attention(const void* q, int q_row_stride, const void* kcache, const void* vcache, const int* block_table,
                            int max_blocks, const int* token_request, const int* positions, void* out, int n_tokens,
                            const Geometry& g, float scale, const float* sink, bool split, bool grouped, int od,
                            long long blocks, cudaStream_t s) {
#define TLLM_ATT_GENERIC(SPLIT_, OD_)                                                                                  \
  TLLM_LAUNCH("paged_attention_generic", (paged_attention_generic_kernel<T, TO, SPLIT_, OD_>), (unsigned)blocks,       \
              (SPLIT_ ? WAYS : WARPS) * 32, 0, s, (const T*)q, q_row_stride, (const T*)kcache, (const T*)vcache,       \
              block_table, max_blocks, token_request, positions, (TO*)out, n_tokens, g, scale, sink)
#define TLLM_ATT_GROUPED(OD_)                                                                                          \
  TLLM_LAUNCH("paged_attention_grouped", (paged_attention_grouped_kernel<T, TO, OD_>), (unsigned)blocks,               \
              GroupedWarps<OD_>::N * 32, 0, s, (const T*)q, q_row_stride, (const T*)kcache, (const T*)vcache,          \
              block_table, max_blocks, token_request, positions, (TO*)out, n_tokens, g, scale, sink)
  if (split) {
    if (od == 2) TLLM_ATT_GENERIC(true, 2); else if (od == 4) TLLM_ATT_GENERIC(true, 4); else if (od == 8) TLLM_ATT_GENERIC(true, 8);
    else TLLM_ATT_GENERIC(true, 16);
  } else if (grouped) {
    if (od == 2) TLLM_ATT_GROUPED(2); else if (od == 4) TLLM_ATT_GROUPED(4); else TLLM_ATT_GROUPED(8);
  } else {
    if (od == 2) TLLM_ATT_GENERIC(false, 2); else if (od == 4) TLLM_ATT_GENERIC(false, 4); else TLLM_ATT_GENERIC(false, 8);
  }
#undef TLLM_ATT_GROUPED
#undef TLLM_ATT_GENERIC
  return TLLM_OK;
}

}  // namespace tllm

using namespace tllm;

// Attention with `maps` score maps per head and key rows of `kd`, value rows of `vd` values.  `nq` query heads and
// `nkv` key/value heads; the key cache holds nkv * maps rows per slot, the value cache nkv.  `chunk` > 0: keys are
// visible inside the query's chunk of positions only.  out_f32 != 0: the output rows are float32 whatever the cache's type.
// `sink` (float32, one per query head, or null): exp(sink) joins every softmax's denominator of that head.
// `keep`: the first positions that a window leaves visible; `rel` (float32 [nq, rel_len] or null): a bias per head and
// distance.  `max_q_len`: the most tokens of one request in the step (how many rows share their keys; 0 if unknown);
// `max_kv_len`: the most keys of one request, or more, `n_requests` (0 if unknown): they choose the launch, see attention_route.h.
extern "C" int tllm_paged_attention_maps(const void* q, int q_row_stride, const void* kcache, const void* vcache,
                                         const int* block_table, int max_blocks, const int* token_request,
                                         const int* positions, void* out, int n_tokens, int nq, int nkv, int maps, int kd,
                                         int vd, int page_size, long long k_page_stride, long long k_head_stride,
                                         long long v_page_stride, long long v_head_stride, float scale, int window,
                                         int chunk, int dtype, int out_f32, int split_override, const float* sink,
                                         int keep, const float* rel, int rel_len, int max_q_len, int max_kv_len,
                                         int n_requests, void* stream) {
  TLLM_REQUIRE(n_tokens > 0 && nq > 0 && nkv > 0 && nq % nkv == 0 && maps > 0,
               "attention: %d tokens, %d heads, %d key/value heads (heads must be a multiple of key/value heads)", n_tokens, nq, nkv);
  TLLM_REQUIRE(kd >= 1 && kd <= MAX_KD && vd >= 1 && vd <= MAX_VD,
               "attention: key size %d / value size %d is not built (up to %d / %d)", kd, vd, MAX_KD, MAX_VD);
  TLLM_REQUIRE(page_size > 0 && max_blocks > 0 && window >= 0 && chunk >= 0, "attention: page size %d, %d blocks, window %d, chunk %d", page_size, max_blocks, window, chunk);
  TLLM_REQUIRE(keep >= 0 && (rel == nullptr || rel_len >= 1), "attention: %d kept keys, %d distances of a bias", keep, rel_len);
  const int elem = dtype == TLLM_F32 ? 4 : 2;
  TLLM_REQUIRE(dtype == TLLM_F32 || dtype == TLLM_BF16, "attention: unknown dtype code %d", dtype);
  Geometry g;
  g.kvec = (kd * elem) % 16 == 0 && ((size_t)kcache % 16) == 0 && (k_page_stride * elem) % 16 == 0 && (k_head_stride * elem) % 16 == 0;
  g.nq = nq * maps; g.nk = nkv * maps; g.maps = maps; g.kd = kd; g.vd = vd; g.page_size = page_size; g.window = window;
  g.keep = window > 0 ? keep : 0; g.rel = rel; g.rel_len = rel_len;
  g.chunk = chunk; g.k_page_stride = k_page_stride; g.k_head_stride = k_head_stride; g.v_page_stride = v_page_stride;
  g.v_head_stride = v_head_stride;
  const long long tasks = (long long)n_tokens * g.nq;
  // few pairs (decoded tokens): eight warps per pair; the result is the same to the bit
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    TLLM_FAIL(TLLM_ERR_CUDA, "attention: cannot read the number of SMs");
  // Rows that share their keys: several to a CTA
  const long long all_rows = (long long)n_tokens * (nq / nkv);
  long long keys = max_kv_len;
  if (keys > 0 && window > 0 && keys > (long long)window + g.keep) keys = (long long)window + g.keep;
  if (keys > 0 && chunk > 0 && keys > chunk) keys = chunk;
  const int rows = split_override < 0 ? attention_rows_per_cta(n_tokens, max_q_len, n_requests, keys, g.nq, g.nk, kd > 64 || vd > 64, sms)
                                      : (split_override == 3 ? 16 : (split_override == 4 ? 4 : 0));
  const bool vvec = vd % 4 == 0 && ((size_t)vcache % 16) == 0 && v_page_stride % 4 == 0 && v_head_stride % 4 == 0;
  if (dtype == TLLM_F32 && g.kvec && vvec && kd <= 128 && vd <= 128 && rows > 0) {
    const long long wide = (all_rows + 15) / 16 * g.nk, narrow = (all_rows + 3) / 4 * g.nk;
    const bool r16 = rows == 16;
    TLLM_REQUIRE(narrow <= 2147483647LL, "attention: %lld (token, head) pairs exceed the grid", tasks);
    cudaStream_t s = (cudaStream_t)stream;
#define TLLM_ATT_ROWS(OD_, R_)                                                                                         \
  return launch_rows<OD_, R_>((const float*)q, q_row_stride, (const float*)kcache, (const float*)vcache, block_table,  \
                              max_blocks, token_request, positions, (float*)out, n_tokens, g, scale, sink,             \
                              R_ == 16 ? wide : narrow, s)
    if (kd <= 64 && vd <= 64) { if (r16) TLLM_ATT_ROWS(2, 16); TLLM_ATT_ROWS(2, 4); }
    if (r16) TLLM_ATT_ROWS(4, 16);
    TLLM_ATT_ROWS(4, 4);
#undef TLLM_ATT_ROWS
  }
  // split_override: -1 by the number of pairs; 3 and 4: 16 and 4 rows that share their keys (where the sizes allow it); 1 eight warps per pair; 0 one warp per (token, key row, four query rows);
  // 2 one warp per pair (the plainest form, kept for comparison: all give the same bits)
  const bool large = kd > MAX_HD || vd > MAX_HD;
  const bool split = large || (split_override >= 0 ? split_override == 1 : tasks <= 8LL * sms);
  const bool grouped = !split && split_override != 2;
  const int hd = kd > vd ? kd : vd;
  const int od = large ? 16 : (hd <= 64 ? 2 : (hd <= 128 ? 4 : 8));
  const int gw = od <= 2 ? 4 : (od <= 4 ? 2 : 1);
  const long long gtasks = (long long)n_tokens * g.nk * ((nq / nkv + GH - 1) / GH);
  const long long blocks = split ? tasks : (grouped ? (gtasks + gw - 1) / gw : (tasks + WARPS - 1) / WARPS);
  TLLM_REQUIRE(blocks <= 2147483647LL, "attention: %lld (token, head) pairs exceed the grid", tasks);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == TLLM_F32)
    return launch_attention<float, float>(q, q_row_stride, kcache, vcache, block_table, max_blocks, token_request, positions, out,
                                          n_tokens, g, scale, sink, split, grouped, od, blocks, s);
  if (out_f32)
    return launch_attention<__nv_bfloat16, float>(q, q_row_stride, kcache, vcache, block_table, max_blocks, token_request,
                                                  positions, out, n_tokens, g, scale, sink, split, grouped, od, blocks, s);
  return launch_attention<__nv_bfloat16, __nv_bfloat16>(q, q_row_stride, kcache, vcache, block_table, max_blocks, token_request,
                                                        positions, out, n_tokens, g, scale, sink, split, grouped, od, blocks, s);
}

extern "C" int tllm_paged_attention_generic(const void* q, int q_row_stride, const void* kcache, const void* vcache,
                                            const int* block_table, int max_blocks, const int* token_request,
                                            const int* positions, void* out, int n_tokens, int nq, int nkv, int hd,
                                            int page_size, long long page_stride, long long head_stride,
                                            float scale, int window, int dtype, int split_override, int max_q_len,
                                            int max_kv_len, int n_requests, void* stream) {
  TLLM_REQUIRE(hd >= 16 && hd <= MAX_HD && hd % 16 == 0,
               "attention: head size %d is not built (multiples of 16 up to %d are)", hd, MAX_HD);
  const int elem = dtype == TLLM_F32 ? 4 : 2;
  TLLM_REQUIRE(((size_t)vcache % 16) == 0 && (page_stride * elem) % 16 == 0 && (head_stride * elem) % 16 == 0,
               "attention: cache rows must be 16-byte aligned");
  return tllm_paged_attention_maps(q, q_row_stride, kcache, vcache, block_table, max_blocks, token_request, positions, out,
                                   n_tokens, nq, nkv, 1, hd, hd, page_size, page_stride, head_stride, page_stride, head_stride,
                                   scale, window, 0, dtype, 0, split_override, nullptr, 0, nullptr, 0, max_q_len, max_kv_len, n_requests,
                                   stream);
}
