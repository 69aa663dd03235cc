// Grouped-query attention, decode / short-chunk path (dense model family), for sm_100a.
//
//   gqa_rope_kv_write_kernel  rotates q and k in place (half-rotation RoPE on the first rotary_dim
//                             columns of every head, device-computed angles) and scatters k / v rows
//                             into the paged caches [pages, page_tokens, kv_heads, head_dim]
//   gqa_split_mma_kernel      split-KV online-softmax attention: one CTA per (split, kv head, query
//                             row) serves the G = Hq/Hkv query heads that share the kv head
//   gqa_split_kernel          the same with products on the CUDA cores: heads of 256 columns, caches
//                             that do not start on 16 bytes
//   gqa_merge_kernel          log-sum-exp merge of the splits -> [T, Hq*head_dim] bf16
//
// Query rows carry their own position and sequence slot (continuous batching: rows of different
// sequences and prefill chunks share one launch). Reference counterparts: attention_qk_prepare /
// paged_attention_prepare composites (native/src/inferfabric_acl.cpp:1236-1433).
#include <climits>
#include <type_traits>

#include "attn_rule.cuh"
#include "mma16816.cuh"
#include "gemv.cuh"
#include "rope.cuh"
#include "ifab_kernels.h"

using namespace ifab;

namespace {

__device__ __forceinline__ void rope_cs(int pos, int i, int rot, float theta, float* c, float* s) {
  const float inv_freq = exp2f(-(2.f * (float)i / (float)rot) * log2f(theta));
  float sn, cs;
  sincosf((float)pos * inv_freq, &sn, &cs);
  *c = bf16_round(cs);
  *s = bf16_round(sn);
}
__device__ __forceinline__ long row_of(int pos, int slot, const int32_t* page_table, int max_pages, int page_tokens, int num_pages) {
  const int lp = pos / page_tokens;
  if (lp >= max_pages) return -1;
  const int page = page_table[(long)slot * max_pages + lp];
  if (page < 0 || page >= num_pages) return -1;
  return (long)page * page_tokens + (pos % page_tokens);
}

// grid T, 256 threads. Bound by latency (a row is 6 KB): the angles are formed once per pair and not once per head, everything moves in 16-byte
// pieces, and rotated keys go to the row and to the page from registers. 20 heads of 128: 1 row 4.6 -> 2.6 us, 509 rows 9.1 -> 3.9, 2048 rows 17.6 -> 8.2.
__global__ void __launch_bounds__(256) gqa_rope_kv_write_kernel(bf16* qkv, long ld, const int32_t* positions, const int32_t* slots,
                                                                const int32_t* page_table, int max_pages, int page_tokens,
                                                                bf16* k_cache, bf16* v_cache, int num_pages, int Hq, int Hkv, int hd,
                                                                int rot, float theta, uint32_t* status) {
  extern __shared__ __align__(16) float cs[];      // [half] cos, then [half] sin
  grid_dep_launch();
  grid_dep_wait();
  const int t = blockIdx.x;
  const int pos = positions[t];
  if (pos < 0) return;
  bf16* row = qkv + (long)t * ld;
  const int half = rot / 2, kv_elems = Hkv * hd;
  const long r = row_of(pos, slots[t], page_table, max_pages, page_tokens, num_pages);
  if (r < 0 && threadIdx.x == 0 && status) atomicOr(status, IFAB_STATUS_BAD_INDEX);
  bf16 *kdst = k_cache + r * kv_elems, *vdst = v_cache + r * kv_elems;
  const bf16* vsrc = row + (long)(Hq + Hkv) * hd;
  if (r >= 0)
    for (int c = threadIdx.x; c < kv_elems / 8; c += blockDim.x) reinterpret_cast<uint4*>(vdst)[c] = reinterpret_cast<const uint4*>(vsrc)[c];
  for (int i = threadIdx.x; i < half; i += blockDim.x) rope_cs(pos, i, rot, theta, &cs[i], &cs[half + i]);
  __syncthreads();
  if (half % 8 == 0) {
    const int chunks = half / 8;
    for (int i = threadIdx.x; i < (Hq + Hkv) * chunks; i += blockDim.x) {
      const int h = i / chunks, j = (i - h * chunks) * 8;
      bf16* p = row + (long)h * hd + j;
      float a[8], b[8], x[8], y[8];
      unpack8(*reinterpret_cast<const uint4*>(p), a);
      unpack8(*reinterpret_cast<const uint4*>(p + half), b);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float c = cs[j + e], s = cs[half + j + e];
        x[e] = a[e] * c - b[e] * s;
        y[e] = b[e] * c + a[e] * s;
      }
      const uint4 lo = pack8(x), hi = pack8(y);
      *reinterpret_cast<uint4*>(p) = lo;
      *reinterpret_cast<uint4*>(p + half) = hi;
      if (h >= Hq && r >= 0) {
        bf16* k = kdst + (long)(h - Hq) * hd + j;
        *reinterpret_cast<uint4*>(k) = lo;
        *reinterpret_cast<uint4*>(k + half) = hi;
      }
    }
    if (r >= 0 && rot < hd) {        // key columns that do not turn
      const int rest = (hd - rot) / 8;
      for (int i = threadIdx.x; i < Hkv * rest; i += blockDim.x) {
        const long at = (long)(i / rest) * hd + rot + (i % rest) * 8;
        *reinterpret_cast<uint4*>(kdst + at) = *reinterpret_cast<const uint4*>(row + (long)Hq * hd + at);
      }
    }
    return;
  }
  for (int i = threadIdx.x; i < (Hq + Hkv) * half; i += blockDim.x) {
    const int h = i / half, j = i % half;
    bf16* p = row + (long)h * hd;
    const float c = cs[j], s = cs[half + j];
    const float a = __bfloat162float(p[j]), b = __bfloat162float(p[j + half]);
    p[j] = __float2bfloat16_rn(a * c - b * s);
    p[j + half] = __float2bfloat16_rn(b * c + a * s);
  }
  __syncthreads();
  if (r < 0) return;
  const uint4* ksrc = reinterpret_cast<const uint4*>(row + (long)Hq * hd);
  for (int c = threadIdx.x; c < kv_elems / 8; c += blockDim.x) reinterpret_cast<uint4*>(kdst)[c] = ksrc[c];
}

int log2_of(int v) {
  int k = 0;
  while (k < 30 && (1 << k) < v) ++k;
  return v > 0 && (1 << k) == v ? k : -1;
}
struct GqaParams {
  const bf16* q; long ldq; const bf16* k_cache; const bf16* v_cache;
  const int32_t* positions; const int32_t* slots; const int32_t* page_table;
  int max_pages, page_tokens, num_pages;
  float scale; int window;
  int T, Hq, Hkv, kps, max_splits;
  float* scratch;   // [T][Hq][max_splits][HD + 2]
  uint32_t* status;
  const float* sink;                              // [Hq]: exp(sink) joins the softmax denominator of the head; or null
  const bf16* gate; long ldg; int gate_act;       // the result is multiplied by act(gate [T, Hq * HD]); or null
  int gate_head;                                  // the gate has one value per head instead: [T, Hq]
  ScoreRule rule;
  AheadRule ahead;                                // entries that count as the first keys of a row
  float factor;                                   // of the result
  int order;                                      // rows by how much they see
  int group, page_shift, split_shift;             // Hq / Hkv; logarithms of page_tokens and max_splits (-1: none): divisions are most of a short row's start
  // keys of a split of a row that sees n: an even share, at least kps, whole rounds of a CTA (64 keys)
  __device__ __forceinline__ int per_split(int n) const {
    const int share = split_shift >= 0 ? (n + max_splits - 1) >> split_shift : (n + max_splits - 1) / max_splits;
    return (max(kps, share) + 63) / 64 * 64;
  }
};

// what a row sees: entries ahead of its window, then the positions first .. pos
struct Seen {
  int first, ahead, n;
  __device__ __forceinline__ Seen(const GqaParams& p, int pos) : first(first_key(pos, p.window, p.rule.chunked)) {
    ahead = p.ahead.count(first);
    n = ahead + pos + 1 - first;
  }
};
// row of key k of what a row sees; `pooled`: in the caches of the blocks
__device__ __forceinline__ long key_row(const GqaParams& p, const Seen& seen, int k, int slot, bool* pooled) {
  *pooled = k < seen.ahead && p.ahead.pool > 0;
  const int pos = k < seen.ahead ? p.ahead.position(k) : seen.first + k - seen.ahead;
  const long r = row_of(pos, slot, p.page_table, p.max_pages, p.page_tokens, p.num_pages);
  return *pooled && r >= 0 ? r / p.page_tokens * p.ahead.per_page + p.ahead.row(k, p.page_tokens) : r;
}

// HD = head_dim (EPL = HD/32 elements per lane), G = query heads per kv head
template <int HD, int G>
__global__ void __launch_bounds__(256) gqa_split_kernel(GqaParams p) {
  constexpr int EPL = HD / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* sm_acc = reinterpret_cast<float*>(smem_raw);   // [8][G][HD]
  float* sm_m = sm_acc + 8 * G * HD;
  float* sm_l = sm_m + 8 * G;
  grid_dep_launch();
  grid_dep_wait();
  const int split = blockIdx.x, kvh = blockIdx.y, t = blockIdx.z;
  const int pos = p.positions[t];
  if (pos < 0) return;
  const Seen seen(p, pos);
  const int n = seen.n, per = p.per_split(n), k_begin = split * per;
  if (k_begin >= n) return;
  const int k_end = min(n, k_begin + per);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = p.slots[t];
  float qf[G][EPL];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const bf16* qh = p.q + (long)t * p.ldq + (long)(kvh * G + g) * HD + lane * EPL;
#pragma unroll
    for (int i = 0; i < EPL; ++i) qf[g][i] = __bfloat162float(qh[i]);
  }
  float m[G], l[G], acc[G][EPL];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m[g] = -INFINITY;
    l[g] = 0.f;
#pragma unroll
    for (int i = 0; i < EPL; ++i) acc[g][i] = 0.f;
  }
  const int kv_elems = p.Hkv * HD;
  constexpr int KB = 4;
  for (int kb = k_begin + warp; kb < k_end; kb += 8 * KB) {
    float kf[KB][EPL], vf[KB][EPL];
    bool ok[KB];
#pragma unroll
    for (int j = 0; j < KB; ++j) {
      const int k = kb + 8 * j;
      ok[j] = k < k_end;
      if (ok[j]) {
        bool pooled;
        const long r = key_row(p, seen, k, slot, &pooled);
        if (r < 0) {
          if (lane == 0 && p.status) atomicOr(p.status, IFAB_STATUS_BAD_INDEX);
          ok[j] = false;
        } else {
          const bf16* kr = (pooled ? (const bf16*)p.ahead.k : p.k_cache) + r * kv_elems + (long)kvh * HD + lane * EPL;
          const bf16* vr = (pooled ? (const bf16*)p.ahead.v : p.v_cache) + r * kv_elems + (long)kvh * HD + lane * EPL;
#pragma unroll
          for (int i = 0; i < EPL; i += 2) {
            const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(kr + i));
            const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(vr + i));
            kf[j][i] = a.x; kf[j][i + 1] = a.y;
            vf[j][i] = b.x; vf[j][i + 1] = b.y;
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < KB; ++j) {
      if (!ok[j]) continue;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < EPL; ++i) s = fmaf(qf[g][i], kf[j][i], s);
        s = warp_sum(s) * p.scale;
        if (!p.rule.plain()) s = ruled_score<true>(s, p.rule, p.rule.slopes ? p.rule.slopes[kvh * G + g] : 0.f, n - 1 - (kb + 8 * j));
        const float mn = fmaxf(m[g], s);
        const float corr = __expf(m[g] - mn), pe = __expf(s - mn);
        l[g] = l[g] * corr + pe;
#pragma unroll
        for (int i = 0; i < EPL; ++i) acc[g][i] = acc[g][i] * corr + pe * vf[j][i];
        m[g] = mn;
      }
    }
  }
#pragma unroll
  for (int g = 0; g < G; ++g) {
    if (lane == 0) {
      sm_m[warp * G + g] = m[g];
      sm_l[warp * G + g] = l[g];
    }
#pragma unroll
    for (int i = 0; i < EPL; ++i) sm_acc[((long)warp * G + g) * HD + lane * EPL + i] = acc[g][i];
  }
  __syncthreads();
  for (int g = 0; g < G; ++g) {
    float M = -INFINITY;
    for (int w = 0; w < 8; ++w) M = fmaxf(M, sm_m[w * G + g]);
    float wgt[8], L = 0.f;
    for (int w = 0; w < 8; ++w) {
      wgt[w] = (sm_m[w * G + g] == -INFINITY) ? 0.f : __expf(sm_m[w * G + g] - M);
      L += wgt[w] * sm_l[w * G + g];
    }
    float* out = p.scratch + (((long)t * p.Hq + kvh * G + g) * p.max_splits + split) * (HD + 2);
    for (int c = threadIdx.x; c < HD; c += blockDim.x) {
      float v = 0.f;
      for (int w = 0; w < 8; ++w) v += wgt[w] * sm_acc[((long)w * G + g) * HD + c];
      out[c] = v;
    }
    if (threadIdx.x == 0) {
      out[HD] = M;
      out[HD + 1] = L;
    }
  }
}

// The same on the tensor cores, for heads of 64 or 128 columns and groups of up to eight query heads. A CTA of four or eight warps works on one split of
// one (row, kv head); every warp streams 16 keys and values at a time through a ring of its own in shared memory (cp.async, 16 bytes, no barrier
// among the warps) and keeps a running maximum, sum and output, merged at the end.
//
//   scores   m16n8k16: the group's query rows are rows 0-7 AND 8-15 of A (so both halves of C hold them), keys are columns. Groups of up to four are there
//            twice in each half
//   values   the weights enter as three bf16 terms that hold all of their 24 bits; the sum is f32 and the rows of C that belong to a head are added at the
//            end. Up to four heads: the terms are rows 0-3, 8-11 and 4-7 of one product (a lane has the weights of its row, so it only picks a
//            term). Eight (WIDE): the first two terms are rows 0-7 and 8-15, and in a second product half of the third is in both
//
// Bound by the stream of keys and values while all CTAs run (a tile of 16 keys takes a warp 1100 clocks and about as long again until the next one is there), and by what
// comes before and behind: rows' order, the start's chain of loads (position, page, keys: divisions are shifts, the pages of 32 tiles one trip, the query's columns
// requested behind them) and the merge (a warp a head; parts pushed to the CTA that adds them up, one cluster barrier). 16 query heads over 4: 64 rows of 2560
// keys (335 MB) 376 us on the CUDA cores, 96 before these, 75 now (4.5 TB/s); 64 rows of 1250, 32 heads 65 -> 49; one row of 2000 keys 10.8 -> 8.0, of
// 4000 16.2 -> 11.0; 8 rows of 1900 15.7 -> 15.5. A third stage of keys or a third CTA an SM gave nothing.
// WITHIN, TWO: where pages hold a multiple of 16 positions a tile is rows that lie one behind the other in one page, with no masks inside; behind a window that begins
// inside sixteen positions, the last of one page's and the first of the next one's (a form of its own: the choice of a page cost the others 0.3 us, one row of
// 1000 keys 8.6 us and 8.3, 28 of 4000 keys 19.1 and 18.7). (Tiles from a multiple of sixteen on counted up to 15 keys more than the window has, a tile
// more and, in whole rounds of a CTA, up to twice the share: windows of 512, eight splits, four rows of four kv heads 7.7 us so, 6.9 now, six 8.2 and 7.0.)
// Every product of sixteen is added to its f32 sum outside the tensor core, scores in two sums each: the tensor core cuts off what it adds up, and chains of its
// products left results 0.6e-6 to 1.9e-6 off, where these are 2.5e-7 to 4.2e-7 and FMAs 2.4e-7 to 4.4e-7. Against two terms of a weight and chains: 64 rows of up
// to 4096 keys 91.2 -> 92.8 us; groups of eight (over one kv head) 32.9 -> 35.0 us.
// Where a tile's sixteen keys lie: each by itself (ANY), one behind the other in a page (WITHIN), or the first ones at the end of a page and the others in another (TWO)
enum class Tiles { ANY, WITHIN, TWO };
template <int HD, int W>
struct MmaSplit {
  static constexpr int KEYS = 16, WARPS = W, STAGES = 2, CH = HD / 8;      // CH: 16-byte chunks of a row
  static constexpr int ROW = HD * 2, STAGE = 2 * KEYS * ROW;
  static constexpr int RINGS = WARPS * STAGES * STAGE, SMEM = RINGS + (8 * HD + 8 * 8 * 2) * 4;
};
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_addr(const float* mine, uint32_t rank) {
  uint32_t at;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_addr(mine)), "r"(rank));
  return at;
}
__device__ __forceinline__ void st_peer4(float* mine, uint32_t rank, const float4& v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(peer_addr(mine, rank)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void st_peer2(float* mine, uint32_t rank, float a, float b) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(peer_addr(mine, rank)), "f"(a), "f"(b) : "memory");
}

// CLUSTER: the splits of a (row, kv head) are one cluster (at most eight) and merge their parts over distributed shared memory into `out`; otherwise
// the parts go to the scratch and gqa_merge_kernel follows.
template <int HD, bool CLUSTER, bool WIDE, Tiles TILES, int W>
__global__ void __launch_bounds__(32 * W, HD == 64 ? 16 / W : 8 / W) gqa_split_mma_kernel(GqaParams p, bf16* res, long ldo) {
  using S = MmaSplit<HD, W>;
  constexpr int NT = 32 * W;
  constexpr bool PAGES = TILES != Tiles::ANY, WITHIN = TILES == Tiles::WITHIN;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  grid_dep_launch();
  grid_dep_wait();
  const int split = blockIdx.x, kvh = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int t = blockIdx.z, pos, slot;
  if (p.order) {                   // the rows that see most first: a long one that starts last is what a launch waits for
    __shared__ __align__(16) uint32_t s_key[NT];
    __shared__ int s_row[3];
    const int mine = threadIdx.x < p.T ? p.positions[threadIdx.x] : -1, its = threadIdx.x < p.T ? p.slots[threadIdx.x] : 0;
    const uint32_t key = (uint32_t)(mine < 0 ? 0 : Seen(p, mine).n) << 8 | (255u - threadIdx.x);      // no two alike; at most 256 threads, fewer than 2^23 keys
    s_key[threadIdx.x] = threadIdx.x < p.T ? key : 0;
    __syncthreads();
    int before = 0;
    for (int i = 0; i < (p.T + 3) / 4; ++i) {
      const uint4 k = reinterpret_cast<const uint4*>(s_key)[i];
      before += (k.x > key) + (k.y > key) + (k.z > key) + (k.w > key);
    }
    if (threadIdx.x < p.T && before == t) {
      s_row[0] = threadIdx.x;
      s_row[1] = mine;
      s_row[2] = its;
    }
    __syncthreads();
    t = s_row[0];
    pos = s_row[1];
    slot = s_row[2];
  } else {
    pos = p.positions[t];
    slot = p.slots[t];
  }
  if (pos < 0) return;
  if (CLUSTER) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const Seen seen(p, pos);
  const int n = seen.n, per = p.per_split(n), k_begin = split * per;
  if (!CLUSTER && k_begin >= n) return;
  const int k_end = min(n, k_begin + per);
  const int g = lane >> 2, c2 = (lane & 3) * 2, G = p.group, gh = WIDE ? g : g & 3;      // gh: this lane's head of the group
  const bool ruled = !p.rule.plain();
  const float slope = p.rule.slopes && gh < G ? p.rule.slopes[kvh * G + gh] : 0.f;
  float acc[HD / 8][2], m = -INFINITY, l = 0.f;
#pragma unroll
  for (int i = 0; i < HD / 8; ++i) acc[i][0] = acc[i][1] = 0.f;

  const uint32_t ring = smem_addr(smem_raw) + warp * S::STAGES * S::STAGE;
  const int kv_elems = p.Hkv * HD;
  const int first = k_begin + warp * S::KEYS, stride = S::WARPS * S::KEYS;
  // PAGES (WITHIN and TWO): a tile's positions are base + i * stride on; its keys before `cut` lie in the page of the first of them, the others in that of the last. Behind `pos` is nothing
  const int base = PAGES ? seen.first + first : 0, cut = WITHIN ? 16 : 16 - (base & 15);
  auto there = [&](int i, int key) { return base + i * stride + key <= pos; };
  const int tiles = first < k_end ? (k_end - first + stride - 1) / stride : 0;
  // pages of 32 tiles, one a lane: one trip to memory for all of them
  auto page_of = [&](int i, int key) {
    const int at = base + i * stride + key;
    if (i >= tiles || at > pos) return -1;
    const int lp = p.page_shift >= 0 ? at >> p.page_shift : at / p.page_tokens, page = lp < p.max_pages ? p.page_table[(long)slot * p.max_pages + lp] : -1;
    if (page >= 0 && page < p.num_pages) return page;
    if (p.status) atomicOr(p.status, IFAB_STATUS_BAD_INDEX);
    return -1;
  };
  int page = PAGES ? page_of(lane, 0) : 0, page2 = PAGES && !WITHIN && cut < 16 ? page_of(lane, cut) : page;
  // Where a tile lies. PAGES: its key 0 by the page of the first keys and by that of the others (rows; NOWHERE: no such page). Otherwise key `first + i * stride +
  // (lane & 15)`: 2 * row + (1: among the blocks); -1: nowhere
  constexpr int NOWHERE = INT_MIN;
  struct Rows {
    int a, b;
  };
  using Where = std::conditional_t<PAGES, Rows, long>;
  auto locate = [&](int i) -> Where {
    if constexpr (PAGES) {
      if (i && (i & 31) == 0) {
        page = page_of(i + lane, 0);
        page2 = !WITHIN && cut < 16 ? page_of(i + lane, cut) : page;
      }
      const int at = base + i * stride, its = __shfl_sync(0xffffffffu, page, i & 31), its2 = __shfl_sync(0xffffffffu, page2, i & 31);
      auto in_page = [&](int x) { return p.page_shift >= 0 ? x & (p.page_tokens - 1) : x % p.page_tokens; };
      Rows r{its < 0 ? NOWHERE : its * p.page_tokens + in_page(at), NOWHERE};
      if (WITHIN || cut == 16) r.b = r.a;
      else if (its2 >= 0) r.b = its2 * p.page_tokens + in_page(at + cut) - cut;
      return r;
    } else {
      const int k = first + i * stride + (lane & 15);
      if (k >= k_end) return -1;
      bool pooled;
      const long r = key_row(p, seen, k, slot, &pooled);
      if (r < 0) {
        if (lane < 16 && p.status) atomicOr(p.status, IFAB_STATUS_BAD_INDEX);
        return -1;
      }
      return 2 * r + pooled;
    }
  };
  auto live_key = [&](const Where& where, int i, int key) {
    if constexpr (PAGES) return (WITHIN || key < cut ? where.a : where.b) != NOWHERE && there(i, key);
    else return __shfl_sync(0xffffffffu, where, key) >= 0;
  };
  auto whole_tile = [&](const Where& where, int i) {
    if constexpr (PAGES) return where.a != NOWHERE && (WITHIN || where.b != NOWHERE) && there(i, S::KEYS - 1);
    else return false;
  };
  auto load = [&](int stage, int i, const Where& where) {
    const uint32_t dst0 = ring + stage * S::STAGE;
    const int ch = lane % S::CH;
    if constexpr (PAGES) {
      constexpr int STEP = 32 / S::CH;
      const int key0 = lane / S::CH;
      const int column = kvh * HD + ch * 8;
      const bool whole = whole_tile(where, i);
      if (whole && (WITHIN || where.a == where.b)) {
        const long at = (long)(where.a + key0) * kv_elems + column;
#pragma unroll
        for (int j = 0; j < S::KEYS / STEP; ++j) {
          const int key = key0 + j * STEP;
          const uint32_t dst = dst0 + key * S::ROW + ((ch ^ (key & 7)) << 4);
          copy16(dst, p.k_cache + at + j * STEP * kv_elems, true);
          copy16(dst + S::KEYS * S::ROW, p.v_cache + at + j * STEP * kv_elems, true);
        }
        return;
      }
#pragma unroll
      for (int j = 0; j < S::KEYS / STEP; ++j) {
        const int key = key0 + j * STEP;
        const uint32_t dst = dst0 + key * S::ROW + ((ch ^ (key & 7)) << 4);
        const bool live = whole || live_key(where, i, key);
        const long off = (long)(live ? (WITHIN || key < cut ? where.a : where.b) + key : 0) * kv_elems + column;
        copy16(dst, p.k_cache + off, live);
        copy16(dst + S::KEYS * S::ROW, p.v_cache + off, live);
      }
    }
    if constexpr (!PAGES) {
#pragma unroll
      for (int j = 0; j < S::KEYS * S::CH / 32; ++j) {
        const int key = lane / S::CH + j * (32 / S::CH);
        const long w = __shfl_sync(0xffffffffu, where, key);
        const long at = w < 0 ? 0 : (w >> 1) * kv_elems + (long)kvh * HD + ch * 8;
        const bf16* kb = w >= 0 && (w & 1) ? (const bf16*)p.ahead.k : p.k_cache;
        const bf16* vb = w >= 0 && (w & 1) ? (const bf16*)p.ahead.v : p.v_cache;
        const uint32_t dst = dst0 + key * S::ROW + ((ch ^ (key & 7)) << 4);
        copy16(dst, kb + at, w >= 0);
        copy16(dst + S::KEYS * S::ROW, vb + at, w >= 0);
      }
    }
  };
  Where at[S::STAGES] = {};          // of the tiles in the ring, by stage
#pragma unroll
  for (int i = 0; i < S::STAGES - 1; ++i) {
    if (i < tiles) {
      at[i] = locate(i);
      load(i, i, at[i]);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // query row of head gh: columns 16 i + c2 + {0, 1} and + 8
  uint32_t q[HD / 16][2];
  {
    const bf16* qh = p.q + (long)t * p.ldq + (long)(kvh * G + (gh < G ? gh : 0)) * HD + c2;
    const bool pairs = (reinterpret_cast<uintptr_t>(qh) & 3) == 0;
#pragma unroll
    for (int i = 0; i < HD / 16; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const bf16 *e = qh + 16 * i + 8 * j;
        q[i][j] = gh >= G ? 0u : pairs ? *reinterpret_cast<const uint32_t*>(e) : (uint32_t)__bfloat16_as_ushort(e[0]) | (uint32_t)__bfloat16_as_ushort(e[1]) << 16;
      }
  }
  Where next = locate(S::STAGES - 1);
  for (int i0 = 0; i0 < tiles; i0 += S::STAGES) {
#pragma unroll
    for (int st = 0; st < S::STAGES; ++st) {
      const int i = i0 + st;
      if (i >= tiles) break;
      constexpr int AHEAD = S::STAGES - 1;
      const int to = (st + AHEAD) % S::STAGES;
      if (i + AHEAD < tiles) {
        at[to] = next;
        load(to, i + AHEAD, next);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (i + AHEAD + 1 < tiles) next = locate(i + AHEAD + 1);
      asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD) : "memory");
      __syncwarp();
      const uint32_t kb = ring + st * S::STAGE, vb = kb + S::KEYS * S::ROW;
      uint32_t b[HD / 16][4];
      float s[2][4] = {};                        // [keys c2 .. / c2 + 8 ..][two sums each: of even and of odd pieces of the columns]
#pragma unroll
      for (int kk = 0; kk < HD / 16; ++kk) {       // all of a tile's operands requested together: one after the other their latencies were most of its time
        const int key = (lane >> 4) * 8 + (lane & 7), ch = 2 * kk + ((lane >> 3) & 1);
        ldsm4(kb + key * S::ROW + ((ch ^ (key & 7)) << 4), b[kk]);
      }
#pragma unroll
      for (int kk = 0; kk < HD / 16; ++kk) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float d[4];
          mma16816_alone(d, q[kk][0], q[kk][0], q[kk][1], q[kk][1], b[kk][2 * h], b[kk][2 * h + 1]);
          s[h][2 * (kk & 1)] += d[0];
          s[h][2 * (kk & 1) + 1] += d[1];
        }
      }
#pragma unroll
      for (int j = 0; j < HD / 16; ++j) {
        const int key = ((lane >> 3) & 1) * 8 + (lane & 7), ch = 2 * j + (lane >> 4);
        ldsm4t(vb + key * S::ROW + ((ch ^ (key & 7)) << 4), b[j]);
      }
      // this lane: keys c2, c2 + 1, c2 + 8, c2 + 9 of the tile against head gh
      float w[4];
      float mn = m;
      const bool whole = whole_tile(at[st], i);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = c2 + (j >> 1) * 8 + (j & 1);
        w[j] = (s[j >> 1][j & 1] + s[j >> 1][2 + (j & 1)]) * p.scale;
        if (ruled) w[j] = ruled_score<true>(w[j], p.rule, slope, n - 1 - (first + i * stride + key));
        if (!whole && !live_key(at[st], i, key)) w[j] = -INFINITY;
        mn = fmaxf(mn, w[j]);
      }
      mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
      mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
      if (__any_sync(0xffffffffu, mn > m)) {
        const float corr = mn > m ? __expf(m - mn) : 1.f;
        l *= corr;
#pragma unroll
        for (int j = 0; j < HD / 8; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) acc[j][e] *= corr;
        m = mn;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        w[j] = w[j] == -INFINITY ? LEAST_WEIGHT : weight_of(w[j] - m);
        l += w[j];
      }
      uint32_t lo[3], hi[3];                     // terms of the weights of keys c2, c2 + 1 and of keys c2 + 8, c2 + 9
      three_terms(w[0], w[1], lo, WIDE ? 0.5f : 1.f);
      three_terms(w[2], w[3], hi, WIDE ? 0.5f : 1.f);
      const uint32_t lo0 = WIDE || g < 4 ? lo[0] : lo[2], hi0 = WIDE || g < 4 ? hi[0] : hi[2];
#pragma unroll
      for (int j = 0; j < HD / 16; ++j) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float d[4];
          mma16816_alone(d, lo0, lo[1], hi0, hi[1], b[j][2 * h], b[j][2 * h + 1]);
          if (WIDE) mma16816(d, lo[2], lo[2], hi[2], hi[2], b[j][2 * h], b[j][2 * h + 1]);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            acc[2 * j + h][e] += d[e];
            if (WIDE || g < 4) acc[2 * j + h][e] += d[2 + e];        // rows 12-15 of groups up to four are nobody's
          }
        }
      }
      __syncwarp();            // the stage is read: a later round may overwrite it
    }
  }
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();             // the rings become the warps' results: [WARPS][8][HD], maxima and sums
  float* sm_acc = reinterpret_cast<float*>(smem_raw);
  __shared__ float sm_m[S::WARPS * 8], sm_l[S::WARPS * 8];
  if ((lane & 3) == 0) {
    sm_m[warp * 8 + g] = m;
    sm_l[warp * 8 + g] = l;
  }
#pragma unroll
  for (int j = 0; j < HD / 8; ++j) {
    float2 v = make_float2(acc[j][0], acc[j][1]);
    if (!WIDE) {               // rows 4-7: the third term
      v.x += __shfl_xor_sync(0xffffffffu, v.x, 16);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, 16);
    }
    if (WIDE || g < 4) *reinterpret_cast<float2*>(sm_acc + (warp * 8 + g) * HD + 8 * j + c2) = v;
  }
  __syncthreads();
  // A warp merges a head at a time. CLUSTER: what the warp has goes to the CTA of the cluster that will put the parts of these columns together: its memory behind
  // the rings, [splits][its columns], then maxima and sums [splits][8] (pushed, so that the one barrier is all there is to wait for).
  const int parts = p.max_splits, mine = G * HD / parts;
  float* got = reinterpret_cast<float*>(smem_raw + S::RINGS);
  if (CLUSTER) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");      // all CTAs of the cluster run
  for (int h = warp; h < G; h += S::WARPS) {
    float wgt[S::WARPS], M = -INFINITY, L = 0.f;
#pragma unroll
    for (int w = 0; w < S::WARPS; ++w) {
      wgt[w] = sm_m[w * 8 + h];
      M = fmaxf(M, wgt[w]);
    }
#pragma unroll
    for (int w = 0; w < S::WARPS; ++w) {
      wgt[w] = wgt[w] == -INFINITY ? 0.f : __expf(wgt[w] - M);
      L += wgt[w] * sm_l[w * 8 + h];
    }
    if (lane * 4 < HD) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < S::WARPS; ++w) {
        const float4 a = *reinterpret_cast<const float4*>(sm_acc + (w * 8 + h) * HD + lane * 4);
        v.x += wgt[w] * a.x;
        v.y += wgt[w] * a.y;
        v.z += wgt[w] * a.z;
        v.w += wgt[w] * a.w;
      }
      if (CLUSTER) {
        const int e = h * HD + lane * 4, to = e / mine;
        st_peer4(got + split * mine + e - to * mine, to, v);
      } else {
        float* to = p.scratch + (((long)t * p.Hq + kvh * G + h) * p.max_splits + split) * (HD + 2) + lane * 4;
        to[0] = v.x;
        to[1] = v.y;
        to[2] = v.z;
        to[3] = v.w;
      }
    }
    if (CLUSTER) {
      if (lane < parts) st_peer2(got + G * HD + (split * 8 + h) * 2, lane, M, L);
    } else if (lane == 0) {
      float* to = p.scratch + (((long)t * p.Hq + kvh * G + h) * p.max_splits + split) * (HD + 2) + HD;
      to[0] = M;
      to[1] = L;
    }
  }
  if (!CLUSTER) return;
  cluster_barrier();
  for (int i = threadIdx.x; i < mine; i += NT) {
    const int e = split * mine + i, h = e / HD, c = e - h * HD, head = kvh * G + h;
    float pm[8], pl[8], pv[8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < parts) {
        pm[r] = got[G * HD + (r * 8 + h) * 2];
        pl[r] = got[G * HD + (r * 8 + h) * 2 + 1];
        pv[r] = got[r * mine + i];
      }
    float M = p.sink ? p.sink[head] : -INFINITY;
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < parts) M = fmaxf(M, pm[r]);
    float L = p.sink ? __expf(p.sink[head] - M) : 0.f, v = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < parts && pm[r] != -INFINITY) {
        const float w = __expf(pm[r] - M);
        L += w * pl[r];
        v += w * pv[r];
      }
    v *= L > 0.f ? p.factor / L : 0.f;
    if (p.gate) v *= activate<true>(__bfloat162float(p.gate[(long)t * p.ldg + (p.gate_head ? head : (long)head * HD + c)]), p.gate_act);
    res[(long)t * ldo + (long)head * HD + c] = __float2bfloat16_rn(v);
  }
}

// grid (Hq, T), HD threads
template <int HD>
__global__ void gqa_merge_kernel(GqaParams p, bf16* out, long ldo) {
  __shared__ float wgt[64];
  __shared__ float Ls;
  grid_dep_launch();
  grid_dep_wait();
  const int h = blockIdx.x, t = blockIdx.y;
  const int pos = p.positions[t];
  if (pos < 0) return;
  const int n = Seen(p, pos).n;
  const int per = p.per_split(n), ns = (n + per - 1) / per;
  const float* base = p.scratch + ((long)t * p.Hq + h) * p.max_splits * (HD + 2);
  if (threadIdx.x < 32) {      // up to 64 splits: two per lane
    const int s0 = threadIdx.x, s1 = threadIdx.x + 32;
    const float m0 = s0 < ns ? base[(long)s0 * (HD + 2) + HD] : -INFINITY, m1 = s1 < ns ? base[(long)s1 * (HD + 2) + HD] : -INFINITY;
    const float l0 = s0 < ns ? base[(long)s0 * (HD + 2) + HD + 1] : 0.f, l1 = s1 < ns ? base[(long)s1 * (HD + 2) + HD + 1] : 0.f;
    float M = warp_max(fmaxf(m0, m1));
    if (p.sink) M = fmaxf(M, p.sink[h]);
    const float w0 = m0 == -INFINITY ? 0.f : __expf(m0 - M), w1 = m1 == -INFINITY ? 0.f : __expf(m1 - M);
    wgt[s0] = w0;
    wgt[s1] = w1;
    const float L = warp_sum(w0 * l0 + w1 * l1) + (p.sink ? __expf(p.sink[h] - M) : 0.f);
    if (threadIdx.x == 0) Ls = L;
  }
  __syncthreads();
  const float invL = Ls > 0.f ? p.factor / Ls : 0.f;
  for (int c = threadIdx.x; c < HD; c += blockDim.x) {
    float v = 0.f;
    for (int s = 0; s < ns; ++s) v += wgt[s] * base[(long)s * (HD + 2) + c];
    v *= invL;
    if (p.gate) v *= activate<true>(__bfloat162float(p.gate[(long)t * p.ldg + (p.gate_head ? h : (long)h * HD + c)]), p.gate_act);
    out[(long)t * ldo + (long)h * HD + c] = __float2bfloat16_rn(v);
  }
}

template <int HD>
int launch_merge(const GqaParams& p, bf16* out, long ldo, cudaStream_t s) {
  return launch_chain(gqa_merge_kernel<HD>, dim3(p.Hq, p.T), dim3(HD < 128 ? 64 : 128), 0, s, p, out, ldo);
}
template <int HD, int G>
int launch_gqa(const GqaParams& p, bf16* out, long ldo, cudaStream_t s) {
  const size_t smem = (size_t)(8 * G * HD + 16 * G) * sizeof(float);
  auto k = gqa_split_kernel<HD, G>;
  if (int rc = opt_in_smem(k, smem)) return rc;
  dim3 grid(p.max_splits, p.Hkv, p.T);
  if (int rc = launch_chain(k, grid, dim3(256), smem, s, p)) return rc;
  return launch_merge<HD>(p, out, ldo, s);
}
template <int HD, bool CLUSTER, bool WIDE, Tiles PAGES, int W>
int launch_split(const GqaParams& p, bf16* out, long ldo, cudaStream_t s) {
  constexpr int smem = MmaSplit<HD, W>::SMEM;
  const dim3 grid(p.max_splits, p.Hkv, p.T);
  auto k = gqa_split_mma_kernel<HD, CLUSTER, WIDE, PAGES, W>;
  if (int rc = opt_in_smem(k, smem)) return rc;
  // Balanced: by the device's preference about 30 clusters of eight CTAs ran at once where 33 fit, and the others waited for them. us behind a small launch, 4000 keys: 30 rows 21.5
  // and 18.9, 33 rows 33.0 and 18.9, 8 rows of four kv heads 24.0 and 18.7
  return CLUSTER ? launch_clusters(true, k, grid, dim3(32 * W), (unsigned)p.max_splits, smem, s, p, out, ldo) : launch_chain(k, grid, dim3(32 * W), smem, s, p, out, ldo);
}
template <int HD, bool WIDE, Tiles PAGES>
int launch_mma(const GqaParams& p, bool cluster, int warps, bf16* out, long ldo, cudaStream_t s) {
  if (cluster) return warps == 8 ? launch_split<HD, true, WIDE, PAGES, 8>(p, out, ldo, s) : launch_split<HD, true, WIDE, PAGES, 4>(p, out, ldo, s);
  if (int rc = launch_split<HD, false, WIDE, PAGES, 4>(p, out, ldo, s)) return rc;
  return launch_merge<HD>(p, out, ldo, s);
}

template <int HD>
int dispatch_g(GqaParams p, bf16* out, long ldo, cudaStream_t s) {
  const int G = p.Hq / p.Hkv;
  if (G != 1 && G != 2 && G != 4 && G != 8) return -1;
  // Many rows fill the chip by themselves: then fewer splits, each longer, so that a CTA's start and end and the merge weigh less: as many CTAs as two
  // to an SM. 64 rows of 2560 keys: 77 us with 2 splits, 89 with 4; 27 rows of 1024: 20 us with 2, 35 with 8; 8 rows of 1900: 13 us with 8.
  const int rows = p.T > 0 ? p.T * p.Hkv : 1, asked = p.max_splits, want = (296 + rows - 1) / rows;
  p.max_splits = asked < want ? asked : want;
  if constexpr (HD <= 128) {
    const uintptr_t bits = (uintptr_t)p.k_cache | (uintptr_t)p.v_cache | (p.ahead.pool > 0 ? (uintptr_t)p.ahead.k | (uintptr_t)p.ahead.v : 0);
    if (bits % 16 == 0) {
      // A cluster of up to eight splits merges by itself, which saves the merge's launch. A few rows with long contexts take more splits than that: from
      // about 512 keys in each of eight on, more CTAs are worth the second launch (one row, four kv heads).
      const bool cluster = rows >= 16 || (long)p.kps * asked <= 4096;
      if (cluster) {
        p.max_splits = want >= 8 ? 8 : want >= 4 ? 4 : want >= 2 ? 2 : 1;
        while (p.max_splits > asked) p.max_splits /= 2;
      }
      // Eight warps a CTA where all CTAs have an SM each: half as many tiles one after the other (one row of 4000 keys 16.1 us by four, 11.0 by eight). The clusters have to
      // fit the GPCs at once, 15 of eight such CTAs and 33 of four (4 rows of 1000 keys, four kv heads of two, in sixteen of eight: 11.6 us by eight, 7.9 by four; 34 rows
      // of 300 keys in 34 of four: 10.4 and 7.3).
      const int warps = cluster && rows * p.max_splits <= (p.max_splits == 8 ? 120 : p.max_splits == 4 ? 132 : 148) ? 8 : 4;
      p.split_shift = log2_of(p.max_splits);
      // more CTAs than run at once (two an SM, heads of 64 four): 64 rows of 1000 to 4000 keys, two splits, 94 us in the rows' order, 82 so; 250 to 1000 keys 30.1 and 28.8; short rows cost
      // less than their order (64 rows of four kv heads of 100 keys 15.1 and 16.2)
      p.order = cluster && p.T <= 32 * warps && rows * p.max_splits > (HD == 64 ? 592 : 296) && (long)p.kps * asked > 512 && (long)p.kps * asked < 1 << 23;
      const Tiles tiles = p.page_tokens % 16 || p.ahead.any() ? Tiles::ANY : p.window > 0 ? Tiles::TWO : Tiles::WITHIN;
      if (G == 8)
        return tiles == Tiles::ANY      ? launch_mma<HD, true, Tiles::ANY>(p, cluster, warps, out, ldo, s)
               : tiles == Tiles::WITHIN ? launch_mma<HD, true, Tiles::WITHIN>(p, cluster, warps, out, ldo, s)
                                        : launch_mma<HD, true, Tiles::TWO>(p, cluster, warps, out, ldo, s);
      return tiles == Tiles::ANY      ? launch_mma<HD, false, Tiles::ANY>(p, cluster, warps, out, ldo, s)
             : tiles == Tiles::WITHIN ? launch_mma<HD, false, Tiles::WITHIN>(p, cluster, warps, out, ldo, s)
                                      : launch_mma<HD, false, Tiles::TWO>(p, cluster, warps, out, ldo, s);
    }
  }
  switch (G) {
    case 1: return launch_gqa<HD, 1>(p, out, ldo, s);
    case 2: return launch_gqa<HD, 2>(p, out, ldo, s);
    case 4: return launch_gqa<HD, 4>(p, out, ldo, s);
    default: return launch_gqa<HD, 8>(p, out, ldo, s);
  }
}

}  // namespace

extern "C" int ifab_gqa_rope_kv_write(void* qkv, long ld, const int32_t* positions, const int32_t* slots,
                                      const int32_t* page_table, int max_pages, int page_tokens, void* k_cache, void* v_cache,
                                      int num_pages, int T, int Hq, int Hkv, int head_dim, int rotary_dim, float theta,
                                      uint32_t* status, void* stream) {
  if (head_dim % 8 || rotary_dim % 2 || rotary_dim > head_dim || ld % 8) return -1;
  return launch_chain(gqa_rope_kv_write_kernel, dim3(T), dim3(256), (size_t)rotary_dim * sizeof(float), (cudaStream_t)stream, (bf16*)qkv, ld, positions, slots,
                      page_table, max_pages, page_tokens, (bf16*)k_cache, (bf16*)v_cache, num_pages, Hq, Hkv, head_dim, rotary_dim,
                      theta, status);
}

extern "C" int ifab_gqa_decode_attention(const void* q, long ldq, const void* k_cache, const void* v_cache,
                                         const int32_t* positions, const int32_t* slots, const int32_t* page_table,
                                         int max_pages, int page_tokens, int num_pages, float scale, int T, int Hq, int Hkv,
                                         int head_dim, int keys_per_split, int max_splits, float* scratch,
                                         uint64_t scratch_bytes, void* out, long ldo, uint32_t* status, void* stream) {
  return ifab_gqa_window_attention(q, ldq, k_cache, v_cache, positions, slots, page_table, max_pages, page_tokens, num_pages, scale, 0, 0.f, nullptr, 0, nullptr, nullptr,
                                   0, 0, 0, 0, 0, nullptr, nullptr, 1.f, T, Hq, Hkv, head_dim, keys_per_split, max_splits, scratch, scratch_bytes, out, ldo, status, stream);
}

// The same over the last `window` positions (0: all) or, `chunked`, the query's own stretch of as many; with a cap of the scores (0: none), slopes [Hq]
// of the distance bias, a sink logit per query head in the denominator and an output gate, [T, Hq * HD] or [T, Hq]; entries ahead of the window
// (attn_rule.cuh); a factor on the result.
extern "C" int ifab_gqa_window_attention(const void* q, long ldq, const void* k_cache, const void* v_cache, const int32_t* positions, const int32_t* slots,
                                         const int32_t* page_table, int max_pages, int page_tokens, int num_pages, float scale, int window, float cap,
                                         const float* slopes, int chunked, const float* sink, const void* gate, long ldg, int gate_act, int gate_per_head, int keep, int pool, const void* pool_k,
                                         const void* pool_v, float factor, int T, int Hq, int Hkv, int head_dim,
                                         int keys_per_split, int max_splits, float* scratch, uint64_t scratch_bytes, void* out, long ldo,
                                         uint32_t* status, void* stream) {
  if (Hkv < 1 || Hq % Hkv || max_splits < 1 || max_splits > 64 || keys_per_split < 8 || window < 0 || cap < 0.f) return -1;
  const AheadRule ahead = ahead_rule(keep, pool, pool_k, pool_v, page_tokens);
  if (!ahead_ok(ahead, window, chunked) || (ahead.any() && (cap > 0.f || slopes))) return -1;
  if ((uint64_t)T * Hq * max_splits * (head_dim + 2) * sizeof(float) > scratch_bytes) return -5;
  GqaParams p{(const bf16*)q, ldq, (const bf16*)k_cache, (const bf16*)v_cache, positions, slots, page_table,
              max_pages, page_tokens, num_pages, scale, window, T, Hq, Hkv, keys_per_split, max_splits, scratch, status, sink, (const bf16*)gate, ldg,
              gate_act, gate_per_head, {cap, slopes, chunked}, ahead, factor, 0, Hq / Hkv, log2_of(page_tokens), -1};
  cudaStream_t s = (cudaStream_t)stream;
  switch (head_dim) {
    case 64: return dispatch_g<64>(p, (bf16*)out, ldo, s);
    case 128: return dispatch_g<128>(p, (bf16*)out, ldo, s);
    case 256: return dispatch_g<256>(p, (bf16*)out, ldo, s);
    default: return -1;
  }
}
