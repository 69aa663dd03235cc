// Products of few rows with a weight matrix on tcgen05:  C[M, N] = A[M, K] B[N, K]^T with the epilogue of tc_gemm.cu, for M up to a few hundred
// (decode steps of several sequences, short prompts).
//
// Bound by the stream of B, so the work is split for that: the 128 rows of an MMA are WEIGHT rows (output features), the tokens its columns, and
// the K blocks of a tile are shared by the CTAs of a cluster (up to 8), which makes enough CTAs for every SM - two on each - whatever N and K
// are. Each CTA sums its part in tensor memory, puts it into its own shared memory as f32, and after a cluster barrier every CTA adds up a
// share of the tokens over the cluster's parts (distributed shared memory, always in the order of the parts) and stores it. Against one CTA
// per 32 columns and all of K the tokens' rows are read N / 128 times instead of N / 32 times, and no product is left with fewer CTAs than SMs.
//   8 rows, us before -> after:  N 2048 K 6144 34.0 -> 9.8, N 3072 K 2048 13.0 -> 6.9, N 8192 K 2048 14.0 -> 10.5, gated 2 x 6144 K 2048 19.0 -> 18.0 (43
//   as a grouped product), N 151936 K 2048 118 -> 104
//
// Warp 0 issues the copies (A tiles and weight tiles of 64 columns, 128-byte swizzle), warp 1 the MMAs, warps 2-5 read the accumulator; all six
// take part in the sum. With `fixed` (B is written by no kernel of the stream) the ring's first weight tiles are requested before the wait for
// the preceding kernel: they stream in while that one ends.
// Tensor memory is allocated after that wait and the next kernel admitted after the allocation, so no CTA that holds columns ever waits for a
// grid that still wants some.
// Every wait is bounded. One that runs out raises the CTA's flag and the status word; the warps that read the accumulator then wait for what the CTA has started
// (copies into its ring, products that read it) and leave NaN as their part of the sum, so that the whole tile is NaN.
#include <algorithm>

#include "attn_rule.cuh"
#include "rope.cuh"
#include "tc_gemm_core.cuh"
#include "ifab_kernels.h"

using namespace ifab;
using namespace ifab::tc;

namespace {

constexpr int FT = 128;            // features of a tile (gated: 64 gate rows and their 64 up rows)
constexpr uint32_t DRAIN = 4000000u;   // limit of the waits for what a CTA that gives up has started

template <int TOK>
struct RowsCfg {
  static constexpr int W_BYTES = FT * BK * 2, STAGE = W_BYTES + TOK * BK * 2;
  static constexpr int STAGES = TOK <= 16 ? 6 : TOK <= 32 ? 5 : TOK <= 64 ? 4 : 3;      // two CTAs per SM
  static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
  static constexpr int COLS = TOK < 32 ? 32 : TOK;                                      // of tensor memory
  static_assert(TOK * FT * 4 <= STAGES * STAGE, "the part of the sum takes the ring's place");
};

struct RowsParams {
  void* c; long ldc; int out_f32;
  const bf16* residual; long ldr;
  const float* bias;
  int act; float cap;
  int M, N, K, F;                  // F > 0: gated, N = 2 F
  GatedUnit unit;
  int splits, box;                 // CTAs of a cluster; rows of A's box
  int fixed;
  uint32_t* status; uint32_t spin_limit;
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr, uint32_t rank) {
  uint32_t at;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(addr), "r"(rank));
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
  return v;
}

// four consecutive columns of a row of the result
__device__ __forceinline__ void store4(const RowsParams& p, int row, int col, float (&v)[4], int ncols) {
  const int live = min(4, ncols - col);
  if (live <= 0) return;
  if (!p.F) {
    if (p.bias)
      for (int i = 0; i < live; ++i) v[i] += p.bias[col + i];
    if (p.residual) {
      const bf16* r = p.residual + (long)row * p.ldr + col;
      if (live == 4 && (reinterpret_cast<uintptr_t>(r) & 7) == 0) {
        const uint2 u = *reinterpret_cast<const uint2*>(r);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
        v[0] = bf16_round(v[0]) + a.x;
        v[1] = bf16_round(v[1]) + a.y;
        v[2] = bf16_round(v[2]) + b.x;
        v[3] = bf16_round(v[3]) + b.y;
      } else {
        for (int i = 0; i < live; ++i) v[i] = bf16_round(v[i]) + __bfloat162float(r[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (p.act) v[i] = activate<true>(v[i], p.act);
      if (p.cap > 0.f) v[i] = soft_limit<true>(v[i], p.cap);
    }
  }
  if (p.out_f32) {
    float* out = reinterpret_cast<float*>(p.c) + (long)row * p.ldc + col;
    if (live == 4 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
    else
      for (int i = 0; i < live; ++i) out[i] = v[i];
  } else {
    bf16* out = reinterpret_cast<bf16*>(p.c) + (long)row * p.ldc + col;
    if (live == 4 && (reinterpret_cast<uintptr_t>(out) & 7) == 0) {
      const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
      *reinterpret_cast<uint2*>(out) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    } else {
      for (int i = 0; i < live; ++i) out[i] = __float2bfloat16_rn(v[i]);
    }
  }
}

// grid (feature tiles x splits, token tiles), clusters of `splits` along x
template <int TOK>
__global__ void __launch_bounds__(192) tc_gemm_rows_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, RowsParams p) {
  using C = RowsCfg<TOK>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::STAGES * C::STAGE);
  uint64_t *empty = full + C::STAGES, *acc_full = empty + C::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* requested = abort_flag + 1;      // K blocks whose copies were requested, once no more will be; until then -1
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = blockIdx.x % p.splits, tile = blockIdx.x / p.splits;
  const bool gated = p.F > 0;
  const int n0 = tile * (gated ? FT / 2 : FT), m0 = blockIdx.y * TOK;
  const int blocks = (p.K + BK - 1) / BK, per = (blocks + p.splits - 1) / p.splits;
  const int k0 = part * per, nk = max(0, min(per, blocks - k0));
  const uint32_t bytes = C::W_BYTES + p.box * BK * 2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    *requested = -1;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_w);
  }
  __syncthreads();
  auto load_w = [&](int kb) {
    unsigned char* dst = smem + (kb % C::STAGES) * C::STAGE;
    uint64_t* bar = &full[kb % C::STAGES];
    mbar_expect_tx(bar, bytes);
    tma_load_2d(dst, &tmap_w, bar, (k0 + kb) * BK, n0);
    if (gated) tma_load_2d(dst + C::W_BYTES / 2, &tmap_w, bar, (k0 + kb) * BK, p.F + n0);
  };
  auto load_a = [&](int kb) { tma_load_2d(smem + (kb % C::STAGES) * C::STAGE + C::W_BYTES, &tmap_a, &full[kb % C::STAGES], (k0 + kb) * BK, m0); };
  int ahead = 0;                     // weight tiles requested before the wait
  if (warp == 0 && lane == 0 && p.fixed)
    for (; ahead < min(nk, C::STAGES); ++ahead) load_w(ahead);
  __syncwarp();
  grid_dep_wait();
  if (warp == 0 && lane == 0)
    for (int kb = 0; kb < ahead; ++kb) load_a(kb);
  __syncwarp();
  if (warp == 1) tmem_alloc(tmem_slot, C::COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_dep_launch();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0 && lane == 0) {
    int issued = ahead;
    for (int kb = ahead; kb < nk; ++kb) {
      if (kb >= C::STAGES && !mbar_wait(&empty[kb % C::STAGES], (kb / C::STAGES - 1) & 1, p.spin_limit)) *abort_flag = 1;
      if (*abort_flag) break;
      load_w(kb);
      load_a(kb);
      issued = kb + 1;
    }
    *requested = issued;
    if (*abort_flag && p.status) atomicOr(p.status, IFAB_STATUS_MBAR_TIMEOUT);
  } else if (warp == 1 && lane == 0) {
    constexpr uint32_t idesc = umma_idesc_bf16(FT, TOK);
    for (int kb = 0; kb < nk; ++kb) {
      const int s = kb % C::STAGES;
      if (!mbar_wait(&full[s], (kb / C::STAGES) & 1, p.spin_limit) || *abort_flag) {
        *abort_flag = 1;
        if (p.status) atomicOr(p.status, IFAB_STATUS_MBAR_TIMEOUT);
        break;
      }
      tc_fence_after();
      const uint32_t at = smem_u32(smem + s * C::STAGE);
      const uint64_t dw = umma_desc_sw128(at), da = umma_desc_sw128(at + C::W_BYTES);
#pragma unroll
      for (int k = 0; k < BK / UMMA_K; ++k) umma_bf16(tmem_base, dw + (uint64_t)(2 * k), da + (uint64_t)(2 * k), idesc, kb > 0 || k > 0);
      umma_commit(&empty[s]);
    }
    umma_commit(acc_full);
  }
  __syncwarp();
  // The accumulator complete, all copies have landed and all products have read the ring: it becomes this CTA's part of the sum, [tokens][128].
  float* sum = reinterpret_cast<float*>(smem);
  const int tokens = min(TOK, p.M - m0);
  if (warp >= 2) {
    const bool ready = mbar_wait(acc_full, 0, p.spin_limit);
    tc_fence_after();
    if (!ready) {                    // this limit is for the whole sum, those above are for a block each: either may be the first to run out
      *abort_flag = 1;
      if (lane == 0 && p.status) atomicOr(p.status, IFAB_STATUS_MBAR_TIMEOUT);
    }
    const int f = (warp & 3) * 32 + lane;
    const uint32_t tm = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    if (__any_sync(0xffffffffu, *abort_flag)) {
      for (uint32_t i = 0; i < DRAIN && *requested < 0; ++i) __nanosleep(64);
      const int n = *requested;
      for (int kb = max(0, n - C::STAGES); kb < n; ++kb) mbar_wait(&full[kb % C::STAGES], (kb / C::STAGES) & 1, DRAIN);
      mbar_wait(acc_full, 0, DRAIN);
      for (int t = 0; t < tokens; ++t) sum[t * FT + f] = __int_as_float(0x7fffffff);
    } else {
      for (int c0 = 0; c0 < tokens; c0 += 32) {
        float v[32];
        tmem_ld_32x32(tm + (uint32_t)c0, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (c0 + i < tokens) sum[(c0 + i) * FT + f] = nk > 0 ? v[i] : 0.f;
      }
    }
  }
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, C::COLS);
  const uint32_t sum_at = smem_u32(sum);
  const int groups = gated ? FT / 8 : FT / 4, ncols = gated ? p.F : p.N;
  for (int i = threadIdx.x; ; i += 192) {
    const int t = part + i / groups * p.splits, f = i % groups * 4;
    if (t >= tokens) break;
    float4 v[8], u[8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < p.splits) {
        v[r] = ld_cluster(sum_at + (t * FT + f) * 4, r);
        if (gated) u[r] = ld_cluster(sum_at + (t * FT + FT / 2 + f) * 4, r);
      }
    float a[4] = {v[0].x, v[0].y, v[0].z, v[0].w}, b[4] = {};
    if (gated) b[0] = u[0].x, b[1] = u[0].y, b[2] = u[0].z, b[3] = u[0].w;
#pragma unroll
    for (int r = 1; r < 8; ++r)
      if (r < p.splits) {
        a[0] += v[r].x; a[1] += v[r].y; a[2] += v[r].z; a[3] += v[r].w;
        if (gated) { b[0] += u[r].x; b[1] += u[r].y; b[2] += u[r].z; b[3] += u[r].w; }
      }
    if (gated)
#pragma unroll
      for (int e = 0; e < 4; ++e) a[e] = gated_bf16(a[e], b[e], p.unit);
    store4(p, m0 + t, n0 + f, a, ncols);
  }
  cluster_sync();                    // the parts stay until every CTA has read them
}

int blocks_of(int K) { return (K + BK - 1) / BK; }
// CTAs of a tile's cluster, a power of two (clusters of 3 or 6 leave SMs of a GPC idle: 200 rows, N 3072: 16.9 us by 6, 11.7 by 4), the most that pay:
//   eight K blocks each   while all CTAs run at once, two on an SM. Larger clusters do not pack the GPCs: 256 CTAs by 8 (200 rows, N 2112 K 4096: 272 of them
//                         19.3 us, 136 by 4 16.0), 280 by 4 (384 rows, N 3072 K 2048: 288 of them 21.6, 144 by 2 15.4)
//   six                   by up to 4 (200 rows, N 4096 K 1536: 14.2 us by 2, 11.3 by 4)
//   four                  while every CTA has an SM to itself, by 8 less than half a chip (16 rows, K 2048: N 1024 6.0 us by 4, 5.0 by 8; N 2048 6.2 and 7.0;
//                         K 1024: N 1024 6.3 by 2, 4.5 by 4); from 65 rows on, whose blocks are twice as large, two of them by 8 (128 rows, N 1024 K 1024: 8.1 us
//                         by 4, 7.1 by 8)
int splits_of(int M, int tiles, int blocks) {
  const int sms = device_sms();
  int splits = 8;
  for (; splits > 1; splits /= 2) {
    const long ctas = (long)tiles * splits * 148;
    if ((blocks + splits - 1) / splits * (splits - 1) >= blocks) continue;        // a CTA without work
    if (blocks >= 8 * splits && ctas <= (splits == 8 ? 256 : splits == 4 ? 280 : 296) * sms) break;
    if (blocks >= 6 * splits && splits <= 4 && ctas <= 256 * sms) break;
    if (splits < 8 && blocks >= 4 * splits && ctas <= 148 * sms) break;
    if (splits == 8 && blocks >= (M > 64 ? 2 : 4) * 8 && ctas <= 64 * sms) break;
  }
  return splits;
}

template <int TOK>
int launch(const void* a, long lda, const void* b, long ldb, RowsParams p, cudaStream_t s) {
  auto k = tc_gemm_rows_kernel<TOK>;
  constexpr int smem = RowsCfg<TOK>::SMEM;
  if (int rc = opt_in_smem(k, smem)) return rc;
  p.box = min(TOK, (p.M + 7) / 8 * 8);
  CUtensorMap ta, tw;
  if (int rc = make_tmap_bf16_2d(&ta, a, (uint64_t)p.M, (uint64_t)p.K, (uint64_t)lda, (uint32_t)p.box)) return rc;
  if (int rc = make_tmap_bf16_2d(&tw, b, (uint64_t)p.N, (uint64_t)p.K, (uint64_t)ldb, p.F > 0 ? FT / 2 : FT)) return rc;
  const int tiles = p.F > 0 ? (p.F + FT / 2 - 1) / (FT / 2) : (p.N + FT - 1) / FT, ty = (p.M + TOK - 1) / TOK;
  p.splits = splits_of(p.M, tiles * ty, blocks_of(p.K));
  return launch_chain_cluster(k, dim3(tiles * p.splits, ty), dim3(192), (unsigned)p.splits, (size_t)smem, s, ta, tw, p);
}

}  // namespace

// Whether a product of more than 128 rows is better here than on CTA pairs (tc_gemm_2sm.cu), by what an SM or pair has to load one after the other: a K block is
// 32 KB here, 128 rows of A and half a tile's columns a CTA there, at about 0.37 us per 32 KB in both. From 256 rows on only where that saves eight blocks.
// us here / there: 255 rows 2048 x 6144 16.6 / 34.6, 3072 x 2048 13.1 / 15.3, 8192 x 2048 18.4 / 15.3, 12288 x 2048 29.4 / 19.2; 509 rows 2048 x 6144 19.7 / 34.9,
// 2048 x 2048 13.1 / 14.6, 3072 x 2048 18.3 / 15.7.
bool ifab::tc::rows_better(int M, int N, int K, int F) {
  const int sms = device_sms(), blocks = blocks_of(K), tiles = (F > 0 ? (F + FT / 2 - 1) / (FT / 2) : (N + FT - 1) / FT) * ((M + 127) / 128), splits = splits_of(M, tiles, blocks);
  const long here = (long)((blocks + splits - 1) / splits) * 2 * 256 * std::max(sms, tiles * splits) / sms, there = blocks * pair_loads(M, N);
  return M <= 1024 && there - here >= (M < 256 ? 0 : 8 * 2 * 256);
}

// The caller has checked shapes and strides (tc_gemm.cu); F > 0: gated, N = 2 F. spin_limit: polls of a wait.
extern "C" int ifab_gemm_rows_bf16(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int out_f32, const void* residual, long ldr,
                                   const float* bias, int act, float cap, int unit, float limit, float alpha, int F, int fixed, int M, int N, int K,
                                   uint32_t spin_limit, uint32_t* status, void* stream) {
  if (M < 1 || N < 1 || K < 8 || K % 8 || lda % 8 || ldb % 8 || (F > 0 && N != 2 * F)) return -1;
  RowsParams p{c, ldc, out_f32, (const bf16*)residual, ldr, bias, act, cap, M, N, K, F, {unit, limit, alpha}, 1, 0, fixed, status, spin_limit};
  cudaStream_t s = (cudaStream_t)stream;
  if (M <= 16) return launch<16>(a, lda, b, ldb, p, s);
  if (M <= 32) return launch<32>(a, lda, b, ldb, p, s);
  if (M <= 64) return launch<64>(a, lda, b, ldb, p, s);
  return launch<128>(a, lda, b, ldb, p, s);
}
