// bf16 GEMM on the 5th-generation tensor cores, two-SM form:  C[M,N] = A[M,K] * B[N,K]^T (+ residual), f32 accumulate.
//
// A cluster of two CTAs (a pair of SMs) owns one 256 x 256 output tile. Each CTA streams ITS 128 rows of A and ITS 128 rows
// of B (half of the tile's N) into its own shared memory - 32 KB per 64-wide K block instead of the 48 KB a lone CTA needs for
// a 128 x 256 tile - and the leader CTA issues tcgen05.mma.cta_group::2 (256 x 256 x 16 per instruction), which reads A and B
// from both CTAs' shared memory and accumulates into both CTAs' tensor memory (each CTA keeps its 128 rows x 256 columns).
//
//   warp 0 (both CTAs)   TMA producer: cp.async.bulk.tensor...cta_group::2 into this CTA's stage ring; the bytes of both CTAs
//                        complete on the LEADER's full barrier (its shared::cluster address, by mapa)
//   warp 1 (both CTAs)   allocates tensor memory (cta_group::2, collectively); in the leader one elected lane issues the MMAs and
//                        releases a stage in BOTH CTAs with tcgen05.commit...multicast::cluster
//   warps 2-9 (both)     epilogue of this CTA's 128 rows, two warps for 32 of them: tcgen05.ld, convert, residual, store (tile_rows)
// Six stages of 32 KB, and 4 KB a reader through which its rows pass. No TMA load is multicast: every CTA fetches its own
// tiles. Every mbarrier wait is bounded; a wait that runs out raises the CTA's abort flag and a status bit, and both CTAs still meet at the closing cluster barrier.
// Shapes: N % 32 == 0 (rows are stored 32 columns at a time), K % 8 == 0; M, N and K tails by TMA zero fill and masked stores.
// `ifab_gemm_bf16` uses these kernels from 129 rows and 256 columns up, but where the cluster form has less to load (tc_gemm_rows.cu).
#include <algorithm>

#include "attn_rule.cuh"
#include "rope.cuh"
#include "tc_gemm_core.cuh"
#include "ifab_kernels.h"

using namespace ifab;
using namespace ifab::tc;

namespace {

constexpr int READERS = 8, SLOT_BYTES = 4096, THREADS2 = 64 + 32 * READERS;

// TN: columns of a pair's tile (both CTAs together), also the accumulator's TMEM columns. A CTA supplies TN / 2 rows of B.
template <int TN>
struct Cfg2 {
  static constexpr int HALF_N = TN / 2, STAGES2 = TN == 128 ? 8 : 6;
  static constexpr int A2_BYTES = BM * BK * 2, STAGE2_BYTES = A2_BYTES + HALF_N * BK * 2;
  static constexpr int RING2 = STAGES2 * STAGE2_BYTES;        // then a slot for each reader's rows (tile_rows)
  static constexpr int SMEM2 = RING2 + READERS * SLOT_BYTES + 1024 + 256;
  static constexpr int COLS = TN <= 128 ? 128 : 256;          // an accumulator's share of tensor memory (powers of two)
};

struct Gemm2Params {
  void* c; long ldc; int out_f32;
  const bf16* residual; long ldr;
  int M, N, K;
  uint32_t* status;
  uint32_t spin_limit;
  int staged;     // rows of C (and of the residual) begin on 16 bytes: whole lines by way of shared memory (tile_rows)
  int swiglu_f;   // > 0 (persistent kernel only): B = [gate rows 0..F) | up rows F..2F), C[M, F] = unit(A gate^T, A up^T)
  int act;        // activation of the result (numbers of activate(); 0: none), after bias and residual
  const float* bias; float cap;      // [N] or null; > 0: cap tanh(result / cap)
  GatedUnit unit;
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// the shared::cluster address of the same shared-memory location in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// this CTA's tile -> this CTA's shared memory; completion bytes go to the barrier at `bar_cluster_addr` (the leader's)
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(smem_dst)), "l"(m), "r"(bar_cluster_addr), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}
// arrive on the barrier at this shared-memory offset in BOTH CTAs of the pair once the MMAs issued so far have completed
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3)
               : "memory");
}

__device__ __forceinline__ void add_bias32(const Gemm2Params& p, int col, float* v) {
  if (!p.bias) return;
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] += p.bias[col + i];
}
__device__ __forceinline__ void add_residual8(float* v, const uint4& u) {
  float f[8];
  unpack8(u, f);
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = bf16_round(v[j]) + f[j];
}
__device__ __forceinline__ void finish32(const Gemm2Params& p, float* v) {
  activate_all<true, 32>(v, p.act);
  if (p.cap > 0.f) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = soft_limit<true>(v[i], p.cap);
  }
}
// 32 columns of the lane's own row, straight to C
__device__ __forceinline__ void store_row32_2(const Gemm2Params& p, int row, int col, float* v) {
  if (row >= p.M || col >= (p.swiglu_f > 0 ? p.swiglu_f : p.N)) return;
  add_bias32(p, col, v);
  if (p.residual) {
    const bf16* r = p.residual + (long)row * p.ldr + col;
    if ((reinterpret_cast<uintptr_t>(r) & 15) == 0) {
      uint4 u[4];          // together: one after the other, four trips to L2 for 32 columns (2048 x 2048, K 64, f32 result: 18.3 us, 11.8 so)
#pragma unroll
      for (int i = 0; i < 4; ++i) u[i] = reinterpret_cast<const uint4*>(r)[i];
#pragma unroll
      for (int i = 0; i < 4; ++i) add_residual8(v + 8 * i, u[i]);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = bf16_round(v[i]) + __bfloat162float(r[i]);
    }
  }
  finish32(p, v);
  if (p.out_f32) {
    float* out = reinterpret_cast<float*>(p.c) + (long)row * p.ldc + col;
    if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) reinterpret_cast<float4*>(out)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    } else {
      for (int i = 0; i < 32; ++i) out[i] = v[i];
    }
  } else {
    bf16* out = reinterpret_cast<bf16*>(p.c) + (long)row * p.ldc + col;
    if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) reinterpret_cast<uint4*>(out)[i] = pack8(v + 8 * i);
    } else {
      for (int i = 0; i < 32; ++i) out[i] = __float2bfloat16_rn(v[i]);
    }
  }
}

// The columns a tile has of its row block: [0, width) from n0 on, less at C's edge (both multiples of 32).
__device__ __forceinline__ int tile_cols(const Gemm2Params& p, int n0, int width) { return min(width, (p.swiglu_f > 0 ? p.swiglu_f : p.N) - n0); }

// 16-byte piece `pc` of row `r` in a reader's slot (32 rows x 128 bytes); the rotation keeps both a row's pieces and a column of pieces on all banks
__device__ __forceinline__ uint4* slot_piece(unsigned char* slot, int r, int pc) { return reinterpret_cast<uint4*>(slot) + r * 8 + (pc ^ (r & 7)); }
// requests the residual of 32 rows x `pieces` * 8 columns into the slot, a line a row
__device__ __forceinline__ void request_residual(const Gemm2Params& p, unsigned char* slot, int row0, int col, int pieces, int lane) {
  const int pc = lane & 7;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = 4 * i + (lane >> 3);
    if (row0 + r < p.M && pc < pieces)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(slot_piece(slot, r, pc))), "l"(p.residual + (long)(row0 + r) * p.ldr + col + pc * 8)
                   : "memory");
  }
}
// the residual of the reader's first chunk of a tile, requested while the tile's products still run
__device__ __forceinline__ void request_first(const Gemm2Params& p, unsigned char* slot, int row0, int n0, int width, int half, int lane) {
  const int cols = tile_cols(p, n0, width), c0 = 64 * half;
  if (p.staged && p.residual && c0 < cols) request_residual(p, slot, row0, n0 + c0, min(cols - c0, 64) >> 3, lane);
}

// A reader's part of a tile: 32 rows, every second chunk of 128 bytes of them (`half` 0 or 1: two readers share the 32 lanes of tensor memory a warp can
// reach). A lane holds a row, so its own 16-byte stores touched 32 lines each, half a sector at a time, and with one warp a quarter of tensor memory the
// residual's loads stood in line with them: 4.5 us a tile of 256 x 192 whatever K, 4 us more with a residual. So a finished row goes to the reader's slot, in
// the place its residual was copied to, and leaves it as whole lines, and there are two warps for a quarter. us before -> after, (one warp a quarter):
//   2048 x 2048, residual   K 2048 22.6 -> 19.4 (20.9), K 6144 45.0 -> 41.4 (42.8)      2048 x 3072, K 2048  31.6 -> 28.9 (28.6)
//   1505 x 2048, f32 out    K 2048 18.9 -> 16.6 (16.6), K 6144 40.7 -> 37.8 (38.3)      2048 x (2 x 6144)    83.2 -> 81.8 (81.2; K 64: 34.4 -> 29.8 (35.3))
// The slots take the place of the seventh stage that tiles of 192 columns had, which does not show.
// Direct stores stay for rows that do not begin on 16 bytes, and f32 results with a residual.
template <bool GATED>
__device__ __forceinline__ void tile_rows(const Gemm2Params& p, uint32_t tm_row, int up, unsigned char* slot, int row0, int n0, int width, int half, int lane) {
  if (!p.staged) {
#pragma unroll 1
    for (int c0 = 32 * half; c0 < width; c0 += 64) {
      float v[32];
      tmem_ld_32x32(tm_row + (uint32_t)c0, v);
      if (GATED) {
        float u[32];
        tmem_ld_32x32(tm_row + (uint32_t)(up + c0), u);
        tmem_ld_wait();
        gated_all<32>(v, u, p.unit);
      } else {
        tmem_ld_wait();
      }
      store_row32_2(p, row0 + lane, n0 + c0, v);
    }
    return;
  }
  const int cols = tile_cols(p, n0, width);
  if (!GATED && p.out_f32) {
#pragma unroll 1
    for (int c0 = 32 * half; c0 < cols; c0 += 64) {
      float v[32];
      tmem_ld_32x32(tm_row + (uint32_t)c0, v);
      tmem_ld_wait();
      add_bias32(p, n0 + c0, v);
      finish32(p, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(slot_piece(slot, lane, i)) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
      __syncwarp();
      float* out = reinterpret_cast<float*>(p.c) + n0 + c0 + (lane & 7) * 4;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = 4 * i + (lane >> 3);
        if (row0 + r < p.M) *reinterpret_cast<uint4*>(out + (long)(row0 + r) * p.ldc) = *slot_piece(slot, r, lane & 7);
      }
      __syncwarp();
    }
    return;
  }
#pragma unroll 1
  for (int c0 = 64 * half; c0 < cols; c0 += 128) {
    const int col = n0 + c0, pieces = min(cols - c0, 64) >> 3;
    if (!GATED && p.residual) {
      if (c0 >= 128) request_residual(p, slot, row0, col, pieces, lane);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (4 * h >= pieces) break;
      float v[32];
      tmem_ld_32x32(tm_row + (uint32_t)(c0 + 32 * h), v);
      if (GATED) {
        float u[32];
        tmem_ld_32x32(tm_row + (uint32_t)(up + c0 + 32 * h), u);
        tmem_ld_wait();
        gated_all<32>(v, u, p.unit);
      } else {
        tmem_ld_wait();
      }
      add_bias32(p, col + 32 * h, v);
      if (!GATED && p.residual) {
#pragma unroll
        for (int i = 0; i < 4; ++i) add_residual8(v + 8 * i, *slot_piece(slot, lane, 4 * h + i));
      }
      finish32(p, v);
#pragma unroll
      for (int i = 0; i < 4; ++i) *slot_piece(slot, lane, 4 * h + i) = pack8(v + 8 * i);
    }
    __syncwarp();
    bf16* out = reinterpret_cast<bf16*>(p.c) + col + (lane & 7) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = 4 * i + (lane >> 3);
      if (row0 + r < p.M && (lane & 7) < pieces) *reinterpret_cast<uint4*>(out + (long)(row0 + r) * p.ldc) = *slot_piece(slot, r, lane & 7);
    }
    __syncwarp();
  }
}

// grid (2 * M / 256, N / 256), clusters of 2 along x; THREADS2 threads
template <int TN>
__global__ void __launch_bounds__(THREADS2) tc_gemm_2sm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                                                          Gemm2Params p) {
  using C2 = Cfg2<TN>;
  constexpr int HALF_N = C2::HALF_N, STAGES2 = C2::STAGES2, A2_BYTES = C2::A2_BYTES, STAGE2_BYTES = C2::STAGE2_BYTES;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* slots = smem + C2::RING2;
  uint64_t* full = reinterpret_cast<uint64_t*>(slots + READERS * SLOT_BYTES);
  uint64_t* empty = full + STAGES2;
  uint64_t* acc_full = empty + STAGES2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();       // 0 = leader
  const int m0 = (int)(blockIdx.x >> 1) * 2 * BM + (int)rank * BM;
  const int n0 = (int)blockIdx.y * TN;
  const int num_kb = (p.K + BK - 1) / BK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES2; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, C2::COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                            // the peer's barriers and tensor memory exist before anything is signalled or issued
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dep_launch();
  grid_dep_wait();
  if (warp == 0 && lane == 0) {
    // ---- producer (both CTAs) ----
    int issued = 0;
    for (int kb = 0; kb < num_kb; ++kb) {
      const int s = kb % STAGES2;
      const uint32_t round = kb / STAGES2;
      if (round > 0 && !mbar_wait(&empty[s], (round - 1) & 1, p.spin_limit)) { *abort_flag = 1; break; }
      if (*abort_flag) break;
      unsigned char* a_dst = smem + s * STAGE2_BYTES;
      if (rank == 0) mbar_expect_tx(&full[s], 2 * STAGE2_BYTES);        // this CTA's tiles and the peer's
      const uint32_t bar = map_to_cta(smem_u32(&full[s]), 0);
      tma_load_2d_pair(a_dst, &tmap_a, bar, kb * BK, m0);
      tma_load_2d_pair(a_dst + A2_BYTES, &tmap_b, bar, kb * BK, n0 + (int)rank * HALF_N);
      issued = kb + 1;
    }
    if (*abort_flag && p.status) atomicOr(p.status, IFAB_STATUS_MBAR_TIMEOUT);
    (void)issued;
  } else if (warp == 1 && lane == 0 && rank == 0) {
    // ---- MMA issuer (leader only) ----
    constexpr uint32_t idesc = umma_idesc_bf16(2 * BM, TN);
    bool ok = true;
    for (int kb = 0; kb < num_kb && ok; ++kb) {
      const int s = kb % STAGES2;
      if (!mbar_wait(&full[s], (kb / STAGES2) & 1, p.spin_limit) || *abort_flag) { ok = false; break; }
      tc_fence_after();
      const uint32_t a_addr = smem_u32(smem + s * STAGE2_BYTES);
      const uint64_t da = umma_desc_sw128(a_addr), db = umma_desc_sw128(a_addr + A2_BYTES);
#pragma unroll
      for (int k = 0; k < BK / UMMA_K; ++k) umma_bf16_pair(tmem_base, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, kb > 0 || k > 0);
      umma_commit_pair(&empty[s]);               // frees the stage in both CTAs
    }
    if (!ok) {
      *abort_flag = 1;
      if (p.status) atomicOr(p.status, IFAB_STATUS_MBAR_TIMEOUT);
    }
    umma_commit_pair(acc_full);                  // both CTAs' accumulators are complete (or abandoned)
  } else if (warp >= 2) {
    // ---- epilogue (both CTAs): this CTA's 128 rows ----
    const int q = warp & 3, half = (warp - 2) >> 2, row0 = m0 + q * 32;
    unsigned char* slot = slots + (warp - 2) * SLOT_BYTES;
    request_first(p, slot, row0, n0, TN, half, lane);
    const bool ready = mbar_wait(acc_full, 0, p.spin_limit);
    tc_fence_after();
    if (!ready) {
      *abort_flag = 1;
      if (lane == 0 && p.status) atomicOr(p.status, IFAB_STATUS_MBAR_TIMEOUT);
    }
    if (ready && !*abort_flag) tile_rows<false>(p, tmem_base + ((uint32_t)(q * 32) << 16), 0, slot, row0, n0, TN, half, lane);
    else asm volatile("cp.async.wait_all;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                            // nobody reads the peer's shared or tensor memory any more
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, C2::COLS);
  }
}

// ---- persistent form -------------------------------------------------------------------------------------------------------
// One CTA pair per SM pair (at most 74 pairs) walks the 256 x 256 tiles round-robin. Tensor memory holds TWO accumulators
// (2 x 256 columns = all 512): while the epilogue warps of both CTAs drain tile j, the leader already issues the MMAs of tile
// j + 1 into the other half, and the producers keep the stage ring full across tile boundaries. An accumulator half goes back
// to the issuer when the epilogue warps of both CTAs have arrived on the leader's acc_empty barrier.
// Tile order of the persistent walk: groups of RASTER_M tile rows, inside a group the row index runs fastest. The 74 pairs
// that work at the same time then share a few B tiles (each read by up to RASTER_M pairs back to back) and keep RASTER_M
// tile rows of A in L2, instead of sweeping all of B for every tile row (at 8192^3 B alone is 128 MB - more than L2).
constexpr int RASTER_M = 8;
__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int* tm, int* tn) {
  const int per_group = RASTER_M * tiles_n;
  const int g = t / per_group, within = t - g * per_group;
  const int first = g * RASTER_M, rows = min(RASTER_M, tiles_m - first);
  *tm = first + within % rows;
  *tn = within / rows;
}

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

// grid (2 * pairs), clusters of 2; THREADS2 threads
template <int TN>
__global__ void __launch_bounds__(THREADS2) tc_gemm_2sm_persistent_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                                                                     Gemm2Params p) {
  using C2 = Cfg2<TN>;
  constexpr int HALF_N = C2::HALF_N, STAGES2 = C2::STAGES2, A2_BYTES = C2::A2_BYTES, STAGE2_BYTES = C2::STAGE2_BYTES;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* slots = smem + C2::RING2;
  uint64_t* full = reinterpret_cast<uint64_t*>(slots + READERS * SLOT_BYTES);
  uint64_t* empty = full + STAGES2;
  uint64_t* acc_full = empty + STAGES2;          // [2], one arrival each (the leader's commit, multicast to both CTAs)
  uint64_t* acc_empty = acc_full + 2;            // [2], used in the leader only: an arrival of every epilogue warp of both CTAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
  // SwiGLU mode: a tile is 256 rows x 128 output columns; the leader CTA streams the 128 gate rows of B, its peer the 128
  // matching up rows, so the accumulator holds gate in columns 0..127 and up in 128..255
  const int F = p.swiglu_f;
  const int tiles_n = F > 0 ? (F + HALF_N - 1) / HALF_N : (p.N + TN - 1) / TN, tiles_m = (p.M + 2 * BM - 1) / (2 * BM), tiles = tiles_m * tiles_n;
  const int num_kb = (p.K + BK - 1) / BK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES2; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 2 * READERS);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, 2 * C2::COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dep_launch();
  grid_dep_wait();
  if (warp == 0 && lane == 0) {
    // ---- producer (both CTAs): one ring across all tiles ----
    uint32_t it = 0;
    for (int t = pair; t < tiles && !*abort_flag; t += pairs) {
      int tm, tn;
      tile_coords(t, tiles_m, tiles_n, &tm, &tn);
      const int m0 = tm * 2 * BM + (int)rank * BM, n0 = F > 0 ? tn * HALF_N + (int)rank * F : tn * TN + (int)rank * HALF_N;
      for (int kb = 0; kb < num_kb; ++kb, ++it) {
        const int s = (int)(it % STAGES2);
        const uint32_t round = it / STAGES2;
        if (round > 0 && !mbar_wait(&empty[s], (round - 1) & 1, p.spin_limit)) { *abort_flag = 1; break; }
        if (*abort_flag) break;
        unsigned char* a_dst = smem + s * STAGE2_BYTES;
        if (rank == 0) mbar_expect_tx(&full[s], 2 * STAGE2_BYTES);
        const uint32_t bar = map_to_cta(smem_u32(&full[s]), 0);
        tma_load_2d_pair(a_dst, &tmap_a, bar, kb * BK, m0);
        tma_load_2d_pair(a_dst + A2_BYTES, &tmap_b, bar, kb * BK, n0);
      }
    }
    if (*abort_flag && p.status) atomicOr(p.status, IFAB_STATUS_MBAR_TIMEOUT);
  } else if (warp == 1 && lane == 0 && rank == 0) {
    // ---- MMA issuer (leader only) ----
    constexpr uint32_t idesc = umma_idesc_bf16(2 * BM, TN);
    uint32_t it = 0;
    bool ok = true;
    int j = 0;
    for (int t = pair; t < tiles && ok; t += pairs, ++j) {
      const int b = j & 1;
      // the accumulator half must have been drained by the epilogue of tile j - 2
      if (j >= 2 && !mbar_wait(&acc_empty[b], ((j >> 1) - 1) & 1, p.spin_limit)) { ok = false; break; }
      tc_fence_after();
      const uint32_t d = tmem_base + (uint32_t)(b * C2::COLS);
      for (int kb = 0; kb < num_kb && ok; ++kb, ++it) {
        const int s = (int)(it % STAGES2);
        if (!mbar_wait(&full[s], (it / STAGES2) & 1, p.spin_limit) || *abort_flag) { ok = false; break; }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + s * STAGE2_BYTES);
        const uint64_t da = umma_desc_sw128(a_addr), db = umma_desc_sw128(a_addr + A2_BYTES);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) umma_bf16_pair(d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, kb > 0 || k > 0);
        umma_commit_pair(&empty[s]);
      }
      umma_commit_pair(&acc_full[b]);
    }
    if (!ok) {
      *abort_flag = 1;
      if (p.status) atomicOr(p.status, IFAB_STATUS_MBAR_TIMEOUT);
      // wake the epilogues of both CTAs for every tile they still expect, so that they run into their own bounded waits only once
      for (int b = 0; b < 2; ++b) umma_commit_pair(&acc_full[b]);
    }
  } else if (warp >= 2) {
    // ---- epilogue (both CTAs) ----
    const int q = warp & 3, half = (warp - 2) >> 2;
    unsigned char* slot = slots + (warp - 2) * SLOT_BYTES;
    int j = 0;
    for (int t = pair; t < tiles; t += pairs, ++j) {
      const int b = j & 1;
      int tm, tn;
      tile_coords(t, tiles_m, tiles_n, &tm, &tn);
      const int row0 = tm * 2 * BM + (int)rank * BM + q * 32, n0 = F > 0 ? tn * HALF_N : tn * TN;
      request_first(p, slot, row0, n0, F > 0 ? HALF_N : TN, half, lane);
      const bool ready = mbar_wait(&acc_full[b], (j >> 1) & 1, p.spin_limit);
      tc_fence_after();
      if (!ready || *abort_flag) {
        *abort_flag = 1;
        if (lane == 0 && p.status) atomicOr(p.status, IFAB_STATUS_MBAR_TIMEOUT);
        asm volatile("cp.async.wait_all;" ::: "memory");
        break;
      }
      const uint32_t tm_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * C2::COLS);
      if (F > 0) tile_rows<true>(p, tm_row, HALF_N, slot, row0, n0, HALF_N, half, lane);
      else tile_rows<false>(p, tm_row, 0, slot, row0, n0, TN, half, lane);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty[b]), 0));
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * C2::COLS);
  }
}

bool on_16(const void* rows, long ld, int bytes) { return reinterpret_cast<uintptr_t>(rows) % 16 == 0 && ld * bytes % 16 == 0; }
int pairs_of_device() { return std::max(1, device_sms() / 2); }
// Columns of a tile: of 256, 192 and 128 the width whose waves of tiles over the pairs take least. A K block costs a pair what it loads - 128 rows of A
// and TN / 2 of B in each CTA, about 87 GB/s an SM - rather than what it multiplies, so narrow tiles gain less than their width: 2048 x 3072 (K 2048)
// 32.5 us by 256, 30.3 by 192, 39.7 by 128; 2048 x 8192 56.7, 64.8, 83.6; 1024 x 2048 (K 6144, residual) 42.5, 41.7, 37.8.
int tile_width(int M, int N, int pairs, long* loads = nullptr) {
  int best = 256;
  long least = 0;
  for (int tn : {256, 192, 128}) {
    const long tiles = (long)((M + 255) / 256) * ((N + tn - 1) / tn), cost = (tiles + pairs - 1) / pairs * (256 + tn);
    if (!least || cost < least) least = cost, best = tn;
  }
  if (loads) *loads = least;
  return best;
}
template <int TN>
int launch_2sm(const void* a, long lda, const void* b, long ldb, const Gemm2Params& p, int persistent, int pairs, cudaStream_t s) {
  CUtensorMap ta, tb;
  if (int rc = make_tmap_bf16_2d(&ta, a, (uint64_t)p.M, (uint64_t)p.K, (uint64_t)lda, BM)) return rc;
  if (int rc = make_tmap_bf16_2d(&tb, b, (uint64_t)p.N, (uint64_t)p.K, (uint64_t)ldb, TN / 2)) return rc;
  const int cols = p.swiglu_f > 0 ? (p.swiglu_f + TN / 2 - 1) / (TN / 2) : (p.N + TN - 1) / TN, tiles = (p.M + 255) / 256 * cols;
  constexpr int smem = Cfg2<TN>::SMEM2;
  if (persistent < 0) persistent = tiles > pairs;
  if (!persistent) {
    auto k = tc_gemm_2sm_kernel<TN>;
    if (int rc = opt_in_smem(k, smem)) return rc;
    return launch_chain_cluster(k, dim3(2 * ((p.M + 255) / 256), cols), dim3(THREADS2), 2, (size_t)smem, s, ta, tb, p);
  }
  auto k = tc_gemm_2sm_persistent_kernel<TN>;
  if (int rc = opt_in_smem(k, smem)) return rc;
  return launch_chain_cluster(k, dim3(2 * std::max(1, std::min(tiles, pairs))), dim3(THREADS2), 2, (size_t)smem, s, ta, tb, p);
}
int dispatch_2sm(const void* a, long lda, const void* b, long ldb, const Gemm2Params& p, int persistent, cudaStream_t s) {
  const int pairs = pairs_of_device(), tn = tile_width(p.M, p.N, pairs);
  return tn == 256 ? launch_2sm<256>(a, lda, b, ldb, p, persistent, pairs, s) : tn == 192 ? launch_2sm<192>(a, lda, b, ldb, p, persistent, pairs, s)
                                                                                           : launch_2sm<128>(a, lda, b, ldb, p, persistent, pairs, s);
}

}  // namespace

int ifab::tc::device_sms() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}
long ifab::tc::pair_loads(int M, int N) {
  long loads = 0;
  tile_width(M, N, pairs_of_device(), &loads);
  return loads;
}

// C[M,N] = act(A[M,K] * B[N,K]^T (+ residual)) with CTA pairs on tiles of 256 rows. N % 32 == 0, K % 8 == 0. `persistent` 1: one CTA pair per
// SM pair walks the tiles with two accumulators in tensor memory; 0: one pair per tile; -1: the former where there are more tiles than pairs.
extern "C" int ifab_gemm_act_bf16_2sm(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int out_f32, const void* residual, long ldr,
                                      int act, int persistent, int M, int N, int K, uint32_t* status, void* stream) {
  return ifab_gemm_epilogue_bf16_2sm(a, lda, b, ldb, c, ldc, out_f32, residual, ldr, nullptr, act, 0.f, persistent, M, N, K, status, stream);
}
extern "C" int ifab_gemm_epilogue_bf16_2sm(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int out_f32, const void* residual, long ldr,
                                           const float* bias, int act, float cap, int persistent, int M, int N, int K, uint32_t* status, void* stream) {
  if (M < 1 || N < 32 || N % 32 || K < 8 || K % 8 || lda % 8 || ldb % 8) return -1;
  const int staged = on_16(c, ldc, out_f32 ? 4 : 2) && (!residual || (!out_f32 && on_16(residual, ldr, 2)));
  const Gemm2Params p{c, ldc, out_f32, (const bf16*)residual, ldr, M, N, K, status, 4000000u, staged, 0, act, bias, cap, {}};
  return dispatch_2sm(a, lda, b, ldb, p, persistent, (cudaStream_t)stream);
}
extern "C" int ifab_gemm_bf16_2sm(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int out_f32, const void* residual, long ldr,
                                  int M, int N, int K, uint32_t* status, void* stream) {
  return ifab_gemm_act_bf16_2sm(a, lda, b, ldb, c, ldc, out_f32, residual, ldr, 0, 0, M, N, K, status, stream);
}
extern "C" int ifab_gemm_bf16_2sm_persistent(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int out_f32, const void* residual,
                                             long ldr, int M, int N, int K, uint32_t* status, void* stream) {
  return ifab_gemm_act_bf16_2sm(a, lda, b, ldb, c, ldc, out_f32, residual, ldr, 0, 1, M, N, K, status, stream);
}

extern "C" int ifab_gemm_swiglu_bf16_2sm(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int M, int F, int K, uint32_t* status,
                                         void* stream) {
  return ifab_gemm_gated_bf16_2sm(a, lda, b, ldb, c, ldc, 0, 0.f, 0.f, M, F, K, status, stream);
}
// C[M, F] = unit(A gate^T, A up^T) with B = [gate rows | up rows] ([2F, K]): the packed gate / up projection of a gated feed-forward in
// one persistent CTA-pair launch (gate and up of the same 128 output columns share an accumulator). F % 32 == 0, K % 8 == 0.
extern "C" int ifab_gemm_gated_bf16_2sm(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int unit, float limit, float alpha, int M, int F,
                                        int K, uint32_t* status, void* stream) {
  const GatedUnit gu{unit, limit, alpha};
  if (!gated_ok(gu) || M < 1 || F < 32 || F % 32 || K < 8 || K % 8 || lda % 8 || ldb % 8) return -1;
  const Gemm2Params p{c, ldc, 0, nullptr, 0, M, 2 * F, K, status, 4000000u, on_16(c, ldc, 2), F, 0, nullptr, 0.f, gu};
  return dispatch_2sm(a, lda, b, ldb, p, 1, (cudaStream_t)stream);
}
