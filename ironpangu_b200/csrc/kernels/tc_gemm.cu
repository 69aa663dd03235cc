// bf16 GEMM on the 5th-generation tensor cores:  C[M,N] = A[M,K] * B[N,K]^T (+ residual), f32 accumulate.
//
// One CTA per 128 x BN output tile, three roles:
//   warp 0      TMA producer: streams 128x64 A tiles and BNx64 B tiles (128-byte swizzle) through a
//               ring of shared-memory stages, one mbarrier pair (full / empty) per stage
//   warp 1      allocates tensor memory, then one elected lane issues tcgen05.mma (128 x BN x 16 per
//               instruction, accumulator in TMEM) and releases stages with tcgen05.commit
//   warps 2-5   epilogue: tcgen05.ld the accumulator (each warp its own 32-lane quarter), convert,
//               add the bias / residual, activation or soft limit, store bf16 or f32
// Gated form: B holds gate rows [0, F) and up rows [F, 2 F); a tile's accumulator takes BN / 2 of each (two boxes per stage) and the
// epilogue stores the gated unit's value (rope.cuh), so that a feed-forward's first half is one launch for any number of rows.
// Split form: a product of one tile row with few columns spreads its K over blockIdx.z; its reader adds the parts in their order. Its box of A
// holds the live rows only.
// A and B are both K-major ("NT"), which is how activations [tokens, K] and weights [out, K] are
// stored everywhere in this library, so no transposes are needed. M, N and K tails are handled by
// TMA zero fill plus masked stores. Used where neither tc_gemm_rows.cu (few rows) nor tc_gemm_2sm.cu (CTA pairs, from 129 rows on) is better; the
// reference's counterpart is aclnnMatmul on [T<=4096, K] activations (token_executor.h:387-456).
#include <cstdlib>

#include "attn_rule.cuh"
#include "rope.cuh"
#include "tc_gemm_core.cuh"
#include "ifab_kernels.h"

using namespace ifab;
using namespace ifab::tc;

namespace {

constexpr uint32_t SPIN_LIMIT = 4000000u;       // polls of a wait

struct GemmParams {
  void* c; long ldc; int out_f32;
  const bf16* residual; long ldr;
  int M, N, K;
  uint32_t* status;
  uint32_t spin_limit;
  int a_rows;            // rows of A's box
  int act;               // activation of the result (numbers of activate(); 0: none), after bias and residual
  const float* bias;     // [N] or null
  float cap;             // > 0: the result is cap tanh(result / cap)
  int F; GatedUnit unit; // gated form: output columns (N = 2 F)
  int k_blocks;          // > 0: CTAs of blockIdx.z take that many K blocks each and write f32 parts of the sum, part_stride apart
  long part_stride;
};

// store 32 consecutive columns of one row (values already final)
__device__ __forceinline__ void store_row32(const GemmParams& p, int row, int col, float* v) {
  if (row >= p.M || col >= p.N) return;
  const int nvalid = min(32, p.N - col);
  if (p.bias)
    for (int i = 0; i < nvalid; ++i) v[i] += p.bias[col + i];
  if (p.residual) {
    const bf16* r = p.residual + (long)row * p.ldr + col;
    for (int i = 0; i < nvalid; ++i) v[i] = bf16_round(v[i]) + __bfloat162float(r[i]);
  }
  activate_all<true, 32>(v, p.act);
  if (p.cap > 0.f) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = soft_limit<true>(v[i], p.cap);
  }
  if (p.out_f32) {
    float* out = reinterpret_cast<float*>(p.c) + (long)row * p.ldc + col;
    if (nvalid == 32 && ((reinterpret_cast<uintptr_t>(out) & 15) == 0)) {
#pragma unroll
      for (int i = 0; i < 8; ++i) reinterpret_cast<float4*>(out)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    } else {
      for (int i = 0; i < nvalid; ++i) out[i] = v[i];
    }
  } else {
    bf16* out = reinterpret_cast<bf16*>(p.c) + (long)row * p.ldc + col;
    if (nvalid == 32 && ((reinterpret_cast<uintptr_t>(out) & 15) == 0)) {
#pragma unroll
      for (int i = 0; i < 4; ++i) reinterpret_cast<uint4*>(out)[i] = pack8(v + 8 * i);
    } else {
      for (int i = 0; i < nvalid; ++i) out[i] = __float2bfloat16_rn(v[i]);
    }
  }
}

// 32 consecutive columns of a row of the gated result
__device__ __forceinline__ void store_gated(const GemmParams& p, int row, int col, const float* g, const float* u) {
  if (row >= p.M || col >= p.F) return;
  float v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = gated_bf16(g[i], u[i], p.unit);
  bf16* out = reinterpret_cast<bf16*>(p.c) + (long)row * p.ldc + col;
  const int nvalid = min(32, p.F - col);
  if (nvalid == 32 && ((reinterpret_cast<uintptr_t>(out) & 15) == 0)) {
#pragma unroll
    for (int i = 0; i < 4; ++i) reinterpret_cast<uint4*>(out)[i] = pack8(v + 8 * i);
  } else {
    for (int i = 0; i < nvalid; ++i) out[i] = __float2bfloat16_rn(v[i]);
  }
}

template <int BN, int ST, bool GATED>
__global__ void __launch_bounds__(192) tc_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a,
                                                      const __grid_constant__ CUtensorMap tmap_b, GemmParams p) {
  extern __shared__ unsigned char smem_raw[];
  Pipe<BN, ST> pipe;
  pipe.setup(smem_raw, &tmap_a, &tmap_b);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NOUT = GATED ? BN / 2 : BN;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * NOUT;
  int num_kb = (p.K + BK - 1) / BK, k_first = 0;
  if (p.k_blocks > 0) {
    k_first = blockIdx.z * p.k_blocks;
    num_kb = min(p.k_blocks, num_kb - k_first);
    p.c = reinterpret_cast<float*>(p.c) + blockIdx.z * p.part_stride;
    if (blockIdx.z) p.bias = nullptr;
  }
  grid_dep_launch();
  grid_dep_wait();
  if (warp == 0 && lane == 0) {
    pipe.produce(&tmap_a, &tmap_b, num_kb, m0, n0, -1, p.spin_limit, p.status, GATED ? p.F + n0 : -1, p.a_rows, 0, k_first);
  } else if (warp == 1 && lane == 0) {
    pipe.mma(num_kb, p.spin_limit, p.status);
  } else if (warp >= 2) {
    if (pipe.wait_accumulator(p.spin_limit, p.status)) {
      const int q = warp & 3;                       // TMEM lane quarter this warp may read
      const int row = m0 + q * 32 + lane;
#pragma unroll 1
      for (int c0 = 0; c0 < NOUT; c0 += 32) {
        float v[32];
        tmem_ld_32x32(pipe.tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
        if (GATED) {
          float u[32];
          tmem_ld_32x32(pipe.tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(NOUT + c0), u);
          tmem_ld_wait();
          store_gated(p, row, n0 + c0, v, u);
        } else {
          tmem_ld_wait();
          store_row32(p, row, n0 + c0, v);
        }
      }
    }
  }
  pipe.teardown();
}

template <int BN, int ST, bool GATED = false>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, cudaStream_t s) {
  auto k = tc_gemm_kernel<BN, ST, GATED>;
  constexpr int smem = Cfg<BN, ST>::SMEM;
  if (int rc = opt_in_smem(k, smem)) return rc;
  constexpr int NOUT = GATED ? BN / 2 : BN;
  const int parts = p.k_blocks > 0 ? ((p.K + BK - 1) / BK + p.k_blocks - 1) / p.k_blocks : 1;
  dim3 grid(((GATED ? p.F : p.N) + NOUT - 1) / NOUT, (p.M + BM - 1) / BM, parts);
  return launch_chain(k, grid, dim3(192), (size_t)smem, s, ta, tb, p);
}

}  // namespace

namespace ifab::tc {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

int make_tmap_bf16_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return -20;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld * 2) % 16 || box_rows == 0 || box_rows > 256) return -1;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {64, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -21;
}

int make_tmap_bf16_3d(CUtensorMap* out, const void* base, uint64_t batch, uint64_t rows, uint64_t cols, uint64_t ld,
                      uint64_t bstride, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return -20;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld * 2) % 16 || (bstride * 2) % 16 || box_rows == 0 || box_rows > 256) return -1;
  cuuint64_t dims[3] = {cols, rows, batch};
  cuuint64_t strides[2] = {ld * 2, bstride * 2};
  cuuint32_t box[3] = {64, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -21;
}

}  // namespace ifab::tc

// IFAB_GEMM_2SM=0 keeps every shape on the one-CTA kernel (for A/B timing)
static bool two_sm_enabled() {
  static const bool on = [] {
    const char* v = getenv("IFAB_GEMM_2SM");
    return !(v && v[0] == '0');
  }();
  return on;
}

// C[M,N] = A[M,K] * B[N,K]^T (+ residual). A: row stride lda, B: row stride ldb (elements), K % 8 == 0.
extern "C" int ifab_gemm_bf16(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int out_f32,
                              const void* residual, long ldr, int M, int N, int K, uint32_t* status, void* stream) {
  return ifab_gemm_epilogue_bf16(a, lda, b, ldb, c, ldc, out_f32, residual, ldr, nullptr, 0, 0.f, M, N, K, status, stream);
}

namespace {
// Whether a product of up to 128 rows is better off without shared K, a CTA a tile (its box of A holds the live rows only): a matrix wide enough for an SM a
// tile of 128 columns from `least` rows on (the sum over a cluster is only a detour there: N 151936 K 2048 64 rows 134 us and 127 here, 27 rows 114 and 120; N 32000
// K 1024 64 rows 20.4 and 18.7), and, where the rows are many beside K, one of a quarter of that (N 12288 K 1024 128 rows 15.8 us and 12.6, K 2048 100 rows 19.4 and
// 18.3; N 6144 K 1536 128 rows 12.8 and 12.1, 64 rows 10.6 and 11.3).
bool one_tile_row(int M, int tiles, int K, int least, int per_k = 48) { return tiles > device_sms() ? M > least : 4 * tiles > device_sms() && (long)M * 1024 > (long)per_k * K; }
// columns of its tiles: the narrowest that all run at once, two on an SM
int narrow_tile(int N, int least = 32) {
  int n = least;
  while (n < 128 && (N + n - 1) / n > 2 * device_sms()) n *= 2;
  return n;
}

int gemm_epilogue(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int out_f32, const void* residual, long ldr, const float* bias, int act,
                  float cap, int fixed, int M, int N, int K, uint32_t* status, void* stream) {
  if (M < 1 || N < 1 || K < 8 || K % 8 || lda % 8 || ldb % 8 || cap < 0.f) return -1;
  // Few rows (decode steps, short prompts) are bound by the stream of B: tc_gemm_rows.cu. Above 128 rows by what has to be loaded, and from 256 rows on only for
  // weights: a plain product keeps the order of its sums that the CTA pairs and the one-CTA kernel share.
  const bool alone = M <= BM && one_tile_row(M, (N + 127) / 128, K, 32);
  if (M <= BM ? !alone : (M < 256 || fixed) && rows_better(M, N, K, 0))
    return ifab_gemm_rows_bf16(a, lda, b, ldb, c, ldc, out_f32, residual, ldr, bias, act, cap, 0, 0.f, 0.f, 0, fixed, M, N, K, SPIN_LIMIT, status, stream);
  // CTA pairs (tcgen05.mma cta_group::2; same accumulation order, same bits) - persistent with two accumulators when there is more than one tile per SM
  // pair, one tile per pair otherwise
  if (M > BM && N >= 256 && N % 32 == 0 && two_sm_enabled())
    return ifab_gemm_epilogue_bf16_2sm(a, lda, b, ldb, c, ldc, out_f32, residual, ldr, bias, act, cap, -1, M, N, K, status, stream);
  CUtensorMap ta, tb;
  const int BN = alone ? narrow_tile(N) : N > 128 ? 256 : 128, a_rows = alone ? (M + 7) / 8 * 8 : BM;
  if (int rc = make_tmap_bf16_2d(&ta, a, (uint64_t)M, (uint64_t)K, (uint64_t)lda, (uint32_t)a_rows)) return rc;
  if (int rc = make_tmap_bf16_2d(&tb, b, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, (uint32_t)BN)) return rc;
  GemmParams p{c, ldc, out_f32, (const bf16*)residual, ldr, M, N, K, status, SPIN_LIMIT, a_rows, act, bias, cap, 0, {}, 0, 0};
  cudaStream_t s = (cudaStream_t)stream;
  if (alone) return BN == 32 ? launch<32, 5>(ta, tb, p, s) : BN == 64 ? launch<64, 4>(ta, tb, p, s) : launch<128, 3>(ta, tb, p, s);
  return BN == 256 ? launch<256, 4>(ta, tb, p, s) : launch<128, 6>(ta, tb, p, s);
}

int gemm_gated(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int unit, float limit, float alpha, int fixed, int M, int F, int K,
               uint32_t* status, void* stream) {
  const GatedUnit gu{unit, limit, alpha};
  if (M < 1 || F < 8 || F % 8 || K < 8 || K % 8 || lda % 8 || ldb % 8 || !gated_ok(gu)) return -1;
  const bool alone = M <= BM && one_tile_row(M, (F + 63) / 64, K, 96, 64);      // F 4096 K 1024: 64 rows 8.9 us shared, 9.3 here; 128 rows 11.5 and 10.1
  if (M <= BM ? !alone : (M < 256 || fixed) && rows_better(M, 2 * F, K, F))
    return ifab_gemm_rows_bf16(a, lda, b, ldb, c, ldc, 0, nullptr, 0, nullptr, 0, 0.f, unit, limit, alpha, F, fixed, M, 2 * F, K, SPIN_LIMIT, status, stream);
  if (M > BM && F >= 128 && F % 32 == 0 && two_sm_enabled())
    return ifab_gemm_gated_bf16_2sm(a, lda, b, ldb, c, ldc, unit, limit, alpha, M, F, K, status, stream);
  const int BN = alone ? narrow_tile(2 * F, 64) : 256, a_rows = alone ? (M + 7) / 8 * 8 : BM;
  CUtensorMap ta, tb;
  if (int rc = make_tmap_bf16_2d(&ta, a, (uint64_t)M, (uint64_t)K, (uint64_t)lda, (uint32_t)a_rows)) return rc;
  if (int rc = make_tmap_bf16_2d(&tb, b, (uint64_t)2 * F, (uint64_t)K, (uint64_t)ldb, (uint32_t)(BN / 2))) return rc;
  GemmParams p{c, ldc, 0, nullptr, 0, M, 2 * F, K, status, SPIN_LIMIT, a_rows, 0, nullptr, 0.f, F, gu, 0, 0};
  cudaStream_t s = (cudaStream_t)stream;
  if (alone) return BN == 64 ? launch<64, 4, true>(ta, tb, p, s) : launch<128, 3, true>(ta, tb, p, s);
  return launch<256, 4, true>(ta, tb, p, s);
}
}  // namespace

// The same with a bias [N] in f32 (or null), an activation of the result (rope.cuh) and, for cap > 0, a soft limit of the result (cap tanh(result / cap)) after it.
extern "C" int ifab_gemm_epilogue_bf16(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int out_f32, const void* residual, long ldr,
                                       const float* bias, int act, float cap, int M, int N, int K, uint32_t* status, void* stream) {
  return gemm_epilogue(a, lda, b, ldb, c, ldc, out_f32, residual, ldr, bias, act, cap, 0, M, N, K, status, stream);
}
// The same for a B that no kernel of the stream writes (weights): its first tiles may be read before the preceding kernel has ended.
extern "C" int ifab_gemm_fixed_bf16(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int out_f32, const void* residual, long ldr,
                                    const float* bias, int act, float cap, int M, int N, int K, uint32_t* status, void* stream) {
  return gemm_epilogue(a, lda, b, ldb, c, ldc, out_f32, residual, ldr, bias, act, cap, 1, M, N, K, status, stream);
}

// C[M, F] (bf16) = unit(A gate^T, A up^T) with B = [gate rows | up rows] ([2 F, K]) and the gated units of rope.cuh (0 SiLU, 1 ReLU, 2 limited). F % 8
// == 0. Rows from 129 on go to the CTA pairs where F % 32 == 0 and that is the better form.
extern "C" int ifab_gemm_gated_bf16(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int unit, float limit, float alpha, int M, int F,
                                    int K, uint32_t* status, void* stream) {
  return gemm_gated(a, lda, b, ldb, c, ldc, unit, limit, alpha, 0, M, F, K, status, stream);
}
extern "C" int ifab_gemm_gated_fixed_bf16(const void* a, long lda, const void* b, long ldb, void* c, long ldc, int unit, float limit, float alpha, int M, int F,
                                          int K, uint32_t* status, void* stream) {
  return gemm_gated(a, lda, b, ldb, c, ldc, unit, limit, alpha, 1, M, F, K, status, stream);
}

// Parts of C[M, N] (f32, M <= 128) = A B^T + bias along K: `parts` of them, part_stride elements apart; C is their sum. Every part gets K blocks of 64
// columns, all but the last equally many.
extern "C" int ifab_gemm_split_bf16(const void* a, long lda, const void* b, long ldb, float* c, long ldc, long part_stride, int parts, const float* bias, int M, int N,
                                    int K, uint32_t* status, void* stream) {
  const int kb = (K + BK - 1) / BK, per = parts > 0 ? (kb + parts - 1) / parts : 0;
  if (M < 1 || M > BM || N < 1 || K < 8 || K % 8 || lda % 8 || ldb % 8 || parts < 1 || per * (parts - 1) >= kb || part_stride < (long)(M - 1) * ldc + N) return -1;
  CUtensorMap ta, tb;
  int BN = 32;
  for (; BN < 128 && (N + BN - 1) / BN > 296; BN *= 2) {}
  const int a_rows = (M + 7) / 8 * 8;
  if (int rc = make_tmap_bf16_2d(&ta, a, (uint64_t)M, (uint64_t)K, (uint64_t)lda, (uint32_t)a_rows)) return rc;
  if (int rc = make_tmap_bf16_2d(&tb, b, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, (uint32_t)BN)) return rc;
  GemmParams p{c, ldc, 1, nullptr, 0, M, N, K, status, SPIN_LIMIT, a_rows, 0, bias, 0.f, 0, {}, per, part_stride};
  cudaStream_t s = (cudaStream_t)stream;
  return BN == 128 ? launch<128, 3>(ta, tb, p, s) : BN == 64 ? launch<64, 4>(ta, tb, p, s) : launch<32, 5>(ta, tb, p, s);
}
