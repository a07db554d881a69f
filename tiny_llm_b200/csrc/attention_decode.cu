// bfloat16 attention of decoded tokens over the paged cache: at most 16 rows (new tokens x query heads of the group) per
// request and key/value head, head size 64 or 128 (-DTLLM_HEAD_DIM), no window.
//
// What bounds it is the cache read from memory.  A producer warp walks the block table and fetches a tile of keys and values
// (16 KB: 64 keys of 64 values or 32 of 128) by TMA, a page and a panel of 64 columns per copy and lane, 128-byte
// swizzled; WARPS warps take the tiles in turn, each by itself from scores to P V (mma.sync: the sixteen rows of an item
// leave most of a tcgen05 tile empty), with a running softmax of its own, and meet once at the end.  No barrier per tile,
// and no thread spends its time on copies.  A warp's tiles all pass through one slot of shared memory: were a slot's uses
// other warps' in turn, a warp that waits by parity could take the use before the one in front for its own.  Tiles older
// than the step are asked for before the wait for the launch in front.
//
// `splits` slices of the keys of one (request, key/value head) are a thread-block cluster that merges them over
// distributed shared memory.  Every wait is bounded (status word).
#include <math_constants.h>

#include <map>
#include <mutex>
#include <tuple>

#include "tc_common.cuh"

#ifndef TLLM_HEAD_DIM
#error "compile with -DTLLM_HEAD_DIM=64 or 128"
#endif

TLLM_DEFINE_LAST_ERROR

namespace tllm {

constexpr int HD = TLLM_HEAD_DIM;
static_assert(HD == 64 || HD == 128, "head size 64 or 128");
constexpr int PANELS = HD / 64;              // swizzle rows of 64 values per key
constexpr int TK = 64 / PANELS;              // keys per tile
constexpr int PANEL_BYTES = TK * 128;
constexpr int HALF_BYTES = PANELS * PANEL_BYTES, TILE_BYTES = 2 * HALF_BYTES;   // keys, then values

template <int WARPS_, int CTAS_>
struct Item {
  static constexpr int WARPS = WARPS_, CTAS = CTAS_;               // computing warps = tiles in shared memory; CTAs per SM
  static constexpr int THREADS = WARPS * 32 + 32;                  // ... and the producer
  static constexpr int OFF_MERGE_ML = WARPS * 16 * HD * 4;         // [warp][16 rows][HD], then maxima and sums
  static constexpr int OFF_RESULT = OFF_MERGE_ML + WARPS * 16 * 2 * 4;   // this CTA's result for its cluster [16][HD], then [16][2]
  static constexpr int OFF_BAR = WARPS * TILE_BYTES;
  static constexpr int SMEM = OFF_BAR + 2 * WARPS * 8 + 16 + 1024;       // + alignment slack
  static_assert(OFF_RESULT + 16 * (HD + 2) * 4 <= OFF_BAR, "the merge takes the tiles' place");
};
using Few = Item<4, 3>;     // slices of at most eight tiles
using Many = Item<6, 2>;

struct DecodeParams {
  const __nv_bfloat16* q;
  const int* block_table;   // [R, max_blocks]
  const int* cu_q;          // [R + 1]
  const int* q_start;       // [R]
  __nv_bfloat16* out;       // [T, nq * HD]
  int* status;
  int q_row_stride, max_blocks, nq, nkv, page_size, splits;
  float scale_log2;         // scale * log2(e)
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t* r, uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t* r, uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float2 ld_peer2(const float* ptr, uint32_t rank) {
  uint32_t remote;
  float2 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(ptr)), "r"(rank));
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 16-byte piece `piece` of row `row` of a swizzled tile of keys or values
__device__ __forceinline__ uint32_t piece_at(uint32_t tile, int row, int piece) {
  return tile + (uint32_t)((piece >> 3) * PANEL_BYTES + row * 128 + (((piece & 7) ^ (row & 7)) << 4));
}

template <typename C, bool CLUSTER>
__global__ void __launch_bounds__(C::THREADS, C::CTAS)
attention_decode_tma_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const DecodeParams p) {
  constexpr int WARPS = C::WARPS, RING = WARPS, THREADS = C::THREADS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* empty = full + RING;
  volatile uint32_t* abort_flag = reinterpret_cast<uint32_t*>(empty + RING);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    tma_prefetch_map(&map_k);
    tma_prefetch_map(&map_v);
    for (int s = 0; s < RING; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_trigger();

  // the step's tables are older than the launch in front
  const int req = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z;
  const int group = p.nq / p.nkv;
  const int tok0 = p.cu_q[req], q_len = p.cu_q[req + 1] - tok0, start = p.q_start[req];
  const int rows_total = q_len * group;              // <= 16 by the launch condition
  const int kv_end = start + q_len;
  const int all_tiles = (kv_end + TK - 1) / TK, per_split = (all_tiles + p.splits - 1) / p.splits;
  const int t_begin = split * per_split, n_tiles = max(0, min(all_tiles - t_begin, per_split));
  float* o_sh = reinterpret_cast<float*>(smem);
  float* ml_sh = reinterpret_cast<float*>(smem + C::OFF_MERGE_ML);
  float* c_o = reinterpret_cast<float*>(smem + C::OFF_RESULT);
  float* c_ml = c_o + 16 * HD;

  const int g = lane >> 2, t4 = lane & 3;
  float m_a = -CUDART_INF_F, m_b = -CUDART_INF_F, l_a = 0.f, l_b = 0.f;
  float o[HD / 8][4];
#pragma unroll
  for (int i = 0; i < HD / 8; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }

  if (warp == WARPS) {
    // ---------------- producer: lane = (page of the tile, keys or values, panel)
    const int* table = p.block_table + (size_t)req * p.max_blocks;
    const int pages_per_tile = TK / p.page_size;                       // <= 8: 32 copies at most (head size 128: 4 pages)
    const int pg = lane / (2 * PANELS), panel = lane % PANELS;
    const bool is_v = (lane / PANELS) & 1;
    const uint32_t page_bytes = (uint32_t)p.page_size * HD * 2;
    const CUtensorMap* map = is_v ? &map_v : &map_k;
    const uint32_t off = (is_v ? HALF_BYTES : 0) + panel * PANEL_BYTES + pg * p.page_size * 128;
    const uint64_t once = l2_evict_first_policy();
    auto page_of = [&](int i) {
      const int blk = (t_begin + i) * pages_per_tile + pg;
      return pg < pages_per_tile && i < n_tiles && blk < p.max_blocks && blk * p.page_size < kv_end ? table[blk] : -1;
    };
    int page = page_of(0), i = 0;
    bool waited = false;
    for (; i < n_tiles; ++i) {
      const int s = i % RING;
      const int next = page_of(i + 1);          // (a trip to memory: one tile ahead)
      // a tile that ends before the step's first token is older than the launch in front
      if (!waited && (i >= RING || (t_begin + i + 1) * TK > start)) { pdl_wait(); waited = true; }
      if (i >= RING) {
        bool ok = true;
        if (lane == 0) ok = mbar_wait(&empty[s], ((i / RING) & 1) ^ 1, abort_flag);
        if (!__shfl_sync(0xffffffffu, (int)ok, 0)) {
          if (lane == 0) { *abort_flag = 1; atomicExch(p.status, ERR_AD_PRODUCER); }
          break;
        }
      }
      const int pages = __popc(__ballot_sync(0xffffffffu, page >= 0 && !is_v && panel == 0));
      if (lane == 0) mbar_expect_tx(&full[s], 2u * pages * page_bytes);
      __syncwarp();
      if (page >= 0) tma_load_2d_hint(smem + s * TILE_BYTES + off, map, panel * 64, (page * p.nkv + kvh) * p.page_size, &full[s], once);
      page = next;
    }
    if (lane == 0) mbar_drain(full, RING, i);
    __syncwarp();
  } else {
    // ---------------- this warp's tiles: i = warp, warp + WARPS, ...
    pdl_wait();
    const int pos_a = start + g / group, pos_b = start + (g + 8) / group;
    const bool live_a = g < rows_total, live_b = g + 8 < rows_total;
    const int head_a = kvh * group + g % group, head_b = kvh * group + (g + 8) % group;
    uint32_t qf[HD / 16][4];
    {
      const uint32_t* qa = reinterpret_cast<const uint32_t*>(p.q + (size_t)(tok0 + (live_a ? g / group : 0)) * p.q_row_stride + (size_t)head_a * HD);
      const uint32_t* qb = reinterpret_cast<const uint32_t*>(p.q + (size_t)(tok0 + (live_b ? (g + 8) / group : 0)) * p.q_row_stride + (size_t)head_b * HD);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k) {
        qf[k][0] = live_a ? qa[k * 8 + t4] : 0u;
        qf[k][1] = live_b ? qb[k * 8 + t4] : 0u;
        qf[k][2] = live_a ? qa[k * 8 + 4 + t4] : 0u;
        qf[k][3] = live_b ? qb[k * 8 + 4 + t4] : 0u;
      }
    }
    const float c = p.scale_log2;
    for (int i = warp; i < n_tiles; i += WARPS) {
      const int s = warp;
      const bool ok = mbar_wait(&full[s], (i / RING) & 1, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) { *abort_flag = 1; atomicExch(p.status, ERR_AD_CONSUMER); }
        break;
      }
      const uint32_t kt = smem_u32(smem) + s * TILE_BYTES, vt = kt + HALF_BYTES;
      const int j0 = (t_begin + i) * TK;
      if (j0 + TK > kv_end) {       // rows that hold no key: zeros for values (their weights are zero, and zero times NaN is NaN)
        const int lo = max(0, kv_end - j0);
        for (int idx = lane; idx < (TK - lo) * (HD / 8); idx += 32) {
          const uint32_t at = piece_at(vt, lo + idx / (HD / 8), idx % (HD / 8));
          asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(at), "r"(0u) : "memory");
        }
        __syncwarp();
      }
      // ---- S = Q K^T
      float sc[TK / 8][4];
#pragma unroll
      for (int n = 0; n < TK / 8; ++n) { sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.f; }
#pragma unroll
      for (int k = 0; k < HD / 16; ++k) {
#pragma unroll
        for (int n0 = 0; n0 < TK; n0 += 16) {
          uint32_t b[4];
          ldmatrix_x4(b, piece_at(kt, n0 + (lane & 7) + (lane >> 4) * 8, 2 * k + ((lane >> 3) & 1)));
          mma_bf16(sc[n0 / 8], qf[k], b[0], b[1]);
          mma_bf16(sc[n0 / 8 + 1], qf[k], b[2], b[3]);
        }
      }
      if (j0 + TK - 1 > start) {    // else every row sees all of the tile's keys
#pragma unroll
        for (int n = 0; n < TK / 8; ++n) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = j0 + n * 8 + t4 * 2 + e;
            if (!(live_a && j <= pos_a)) sc[n][e] = -CUDART_INF_F;
            if (!(live_b && j <= pos_b)) sc[n][2 + e] = -CUDART_INF_F;
          }
        }
      }
      float mx_a = -CUDART_INF_F, mx_b = -CUDART_INF_F;
#pragma unroll
      for (int n = 0; n < TK / 8; ++n) {
        mx_a = fmaxf(mx_a, fmaxf(sc[n][0], sc[n][1]));
        mx_b = fmaxf(mx_b, fmaxf(sc[n][2], sc[n][3]));
      }
      mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 1));
      mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 2));
      mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 1));
      mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 2));
      const float mn_a = fmaxf(m_a, mx_a * c), mn_b = fmaxf(m_b, mx_b * c);      // running maxima in scaled (log2) units
      const float ms_a = mn_a == -CUDART_INF_F ? 0.f : mn_a, ms_b = mn_b == -CUDART_INF_F ? 0.f : mn_b;
      const float corr_a = ex2(m_a - ms_a), corr_b = ex2(m_b - ms_b);            // 0 while nothing was seen
      m_a = mn_a; m_b = mn_b;
      uint32_t pf[TK / 16][4];
      float sum_a = 0.f, sum_b = 0.f;
#pragma unroll
      for (int n = 0; n < TK / 8; ++n) {
        const float p0 = ex2(fmaf(sc[n][0], c, -ms_a)), p1 = ex2(fmaf(sc[n][1], c, -ms_a));
        const float p2 = ex2(fmaf(sc[n][2], c, -ms_b)), p3 = ex2(fmaf(sc[n][3], c, -ms_b));
        sum_a += p0 + p1;
        sum_b += p2 + p3;
        pf[n / 2][(n & 1) * 2 + 0] = pack_bf16(p0, p1);
        pf[n / 2][(n & 1) * 2 + 1] = pack_bf16(p2, p3);
      }
      l_a = l_a * corr_a + sum_a;
      l_b = l_b * corr_b + sum_b;
#pragma unroll
      for (int d = 0; d < HD / 8; ++d) { o[d][0] *= corr_a; o[d][1] *= corr_a; o[d][2] *= corr_b; o[d][3] *= corr_b; }
      // ---- O += P V
#pragma unroll
      for (int kk = 0; kk < TK / 16; ++kk) {
#pragma unroll
        for (int d0 = 0; d0 < HD; d0 += 16) {
          uint32_t b[4];
          ldmatrix_x4_trans(b, piece_at(vt, kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, d0 / 8 + (lane >> 4)));
          mma_bf16(o[d0 / 8], pf[kk], b[0], b[1]);
          mma_bf16(o[d0 / 8 + 1], pf[kk], b[2], b[3]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
    }
    l_a += __shfl_xor_sync(0xffffffffu, l_a, 1);
    l_a += __shfl_xor_sync(0xffffffffu, l_a, 2);
    l_b += __shfl_xor_sync(0xffffffffu, l_b, 1);
    l_b += __shfl_xor_sync(0xffffffffu, l_b, 2);
  }

  // ---------------- the warps' running softmaxes meet where the ring was (every copy has landed and been read)
  __syncthreads();
  if (warp < WARPS) {
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) {
      *reinterpret_cast<float2*>(o_sh + (warp * 16 + g) * HD + i * 8 + t4 * 2) = make_float2(o[i][0], o[i][1]);
      *reinterpret_cast<float2*>(o_sh + (warp * 16 + g + 8) * HD + i * 8 + t4 * 2) = make_float2(o[i][2], o[i][3]);
    }
    if (t4 == 0) {
      ml_sh[(warp * 16 + g) * 2] = m_a; ml_sh[(warp * 16 + g) * 2 + 1] = l_a;
      ml_sh[(warp * 16 + g + 8) * 2] = m_b; ml_sh[(warp * 16 + g + 8) * 2 + 1] = l_b;
    }
  }
  __syncthreads();
  for (int idx = tid; idx < rows_total * (HD / 2); idx += THREADS) {
    const int r = idx / (HD / 2), d = (idx % (HD / 2)) * 2;
    float m = -CUDART_INF_F;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) m = fmaxf(m, ml_sh[(w * 16 + r) * 2]);
    const float m_ref = m == -CUDART_INF_F ? 0.f : m;
    float l = 0.f, acc0 = 0.f, acc1 = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float f = exp2f(ml_sh[(w * 16 + r) * 2] - m_ref);   // 0 for a warp that saw no key of the row
      l += f * ml_sh[(w * 16 + r) * 2 + 1];
      const float2 ov = *reinterpret_cast<const float2*>(o_sh + (w * 16 + r) * HD + d);
      acc0 += f * ov.x;
      acc1 += f * ov.y;
    }
    if (CLUSTER) {
      *reinterpret_cast<float2*>(c_o + r * HD + d) = make_float2(acc0, acc1);
      if (d == 0) *reinterpret_cast<float2*>(c_ml + r * 2) = make_float2(m, l);
    } else {
      const size_t th = (size_t)(tok0 + r / group) * p.nq + (size_t)(kvh * group + r % group);
      const float inv = 1.f / l;
      *reinterpret_cast<uint32_t*>(p.out + th * HD + d) = pack_bf16(acc0 * inv, acc1 * inv);
    }
  }
  if (!CLUSTER) return;
  cluster_sync();       // every slice's result lies in its CTA's shared memory; each CTA finishes a share of the elements
  for (int idx = split * THREADS + tid; idx < rows_total * (HD / 2); idx += p.splits * THREADS) {
    const int r = idx / (HD / 2), d = (idx % (HD / 2)) * 2;
    float2 ml[8], ov[8];
    float m = -CUDART_INF_F;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      ml[j] = make_float2(-CUDART_INF_F, 0.f);
      ov[j] = make_float2(0.f, 0.f);
      if (j < p.splits) { ml[j] = ld_peer2(c_ml + r * 2, (uint32_t)j); ov[j] = ld_peer2(c_o + r * HD + d, (uint32_t)j); }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) m = fmaxf(m, ml[j].x);
    const float m_ref = m == -CUDART_INF_F ? 0.f : m;
    float l = 0.f, acc0 = 0.f, acc1 = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float f = exp2f(ml[j].x - m_ref);    // 0 for a slice that saw no key of the row
      l += f * ml[j].y;
      acc0 += f * ov[j].x;
      acc1 += f * ov[j].y;
    }
    const size_t th = (size_t)(tok0 + r / group) * p.nq + (size_t)(kvh * group + r % group);
    const float inv = 1.f / l;
    *reinterpret_cast<uint32_t*>(p.out + th * HD + d) = pack_bf16(acc0 * inv, acc1 * inv);
  }
  cluster_sync();       // no CTA leaves while a peer still reads its shared memory
}

// ---------------------------------------------------------------- host side
// Rows of HD values of a cache, in boxes of one panel of 64 columns x the keys of a page.
static bool make_map_rows(CUtensorMap* map, const void* ptr, long long rows, int box_rows) {
  using Key = std::tuple<const void*, long long, int>;
  static std::map<Key, CUtensorMap> cache;
  static std::mutex mu;
  const Key key(ptr, rows, box_rows);
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if (it != cache.end()) { *map = it->second; return true; }
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)HD, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)HD * 2};
  cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
  cuuint32_t elem[2] = {1, 1};
  if (fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  if (cache.size() > 1024) cache.clear();
  cache[key] = *map;
  return true;
}

}  // namespace tllm

using namespace tllm;

// 1 if the kernel takes these sizes.
extern "C" int tllm_attention_decode_fits(int nq, int nkv, int hd, int page_size, int max_q_len) {
  return hd == HD && nq > 0 && nkv > 0 && nq % nkv == 0 && max_q_len > 0 && (long long)max_q_len * (nq / nkv) <= 16 && page_size >= 8 &&
         page_size <= TK && TK % page_size == 0;
}

namespace tllm {

template <typename C>
static int launch_item(const CUtensorMap& mk, const CUtensorMap& mv, const DecodeParams& p, int n_requests, cudaStream_t s) {
  TLLM_RESERVE_SMEM("attention_decode", C::SMEM, (attention_decode_tma_kernel<C, false>), (attention_decode_tma_kernel<C, true>));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)n_requests, p.nkv, p.splits);
  cfg.blockDim = dim3(C::THREADS);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = p.splits;
  cfg.attrs = pdl_enabled() ? attr : attr + 1;
  cfg.numAttrs = (pdl_enabled() ? 1 : 0) + (p.splits > 1 ? 1 : 0);
  cudaError_t e = p.splits > 1 ? cudaLaunchKernelEx(&cfg, attention_decode_tma_kernel<C, true>, mk, mv, p)
                               : cudaLaunchKernelEx(&cfg, attention_decode_tma_kernel<C, false>, mk, mv, p);
  if (e != cudaSuccess) TLLM_FAIL(TLLM_ERR_CUDA, "attention_decode: %s", cudaGetErrorString(e));
  return TLLM_OK;
}

}  // namespace tllm

// `splits` slices of the keys (1 to 8); `few`: slices of a few tiles, smaller CTAs.
extern "C" int tllm_attention_decode(const void* q, int q_row_stride, const void* kcache, const void* vcache, long long cache_pages,
                                     const int* block_table, int max_blocks, const int* cu_q, const int* q_start, void* out,
                                     int n_requests, int max_q_len, int nq, int nkv, int hd, int page_size, float scale, int splits,
                                     int few, int* status, void* stream) {
  TLLM_REQUIRE(tllm_attention_decode_fits(nq, nkv, hd, page_size, max_q_len), "attention_decode: %d heads, %d key/value heads, head size %d, page size %d, %d tokens "
               "(takes head size %d, at most 16 rows per key/value head, pages of 8 to %d keys)", nq, nkv, hd, page_size, max_q_len, HD, TK);
  TLLM_REQUIRE(n_requests > 0 && max_blocks > 0 && cache_pages > 0 && scale > 0.f && status != nullptr && splits >= 1 && splits <= 8 && nkv <= 65535,
               "attention_decode: %d requests, %d blocks, %lld pages, %d slices", n_requests, max_blocks, cache_pages, splits);
  TLLM_REQUIRE(((uintptr_t)q % 4) == 0 && (q_row_stride % 2) == 0 && ((uintptr_t)kcache % 16) == 0 && ((uintptr_t)vcache % 16) == 0 &&
               ((uintptr_t)out % 4) == 0, "attention_decode: operands are not aligned");
  CUtensorMap mk, mv;
  const long long rows = cache_pages * nkv * page_size;
  TLLM_REQUIRE(rows <= 2147483647LL, "attention_decode: %lld rows in the cache", rows);
  if (!make_map_rows(&mk, kcache, rows, page_size) || !make_map_rows(&mv, vcache, rows, page_size))
    TLLM_FAIL(TLLM_ERR_CUDA, "attention_decode: cuTensorMapEncodeTiled failed");
  DecodeParams p;
  p.q = (const __nv_bfloat16*)q; p.block_table = block_table; p.cu_q = cu_q; p.q_start = q_start; p.out = (__nv_bfloat16*)out;
  p.status = status; p.q_row_stride = q_row_stride; p.max_blocks = max_blocks; p.nq = nq; p.nkv = nkv; p.page_size = page_size;
  p.splits = splits; p.scale_log2 = scale * 1.4426950408889634f;
  return few ? launch_item<Few>(mk, mv, p, n_requests, (cudaStream_t)stream) : launch_item<Many>(mk, mv, p, n_requests, (cudaStream_t)stream);
}
