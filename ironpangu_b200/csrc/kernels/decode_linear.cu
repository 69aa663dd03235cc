// Decode-time (M = 1..8 tokens per tile) linear layers for sm_100a.
//
//   gemv_kernel            y = act(norm(x) W^T) (+ residual)         column-parallel / replicated linears
//   rows_kernel            the same as a stream through rings in shared memory (row_stream.cuh): the dense decoder's linears
//   gemv_allreduce_kernel  y = sum_ranks(x_r W_r^T) + residual       row-parallel linear fused with a
//                          one-shot all-reduce over NVLink peer memory (push partial tiles to every
//                          peer, bounded flag wait, rank-ordered f32 sum) - no separate collective launch
//
// Counterparts in the reference: `linear` + `allreduce` instructions executed by aclnnMatmul and
// HcclAllReduce (native/src/token_executor.h:374-404); here both are one kernel.
#include "gemv.cuh"
#include "oneshot_ar.cuh"
#include "row_stream.cuh"
#include "tc_common.cuh"
#include "ifab_kernels.h"

using namespace ifab;

namespace {

struct GemvParams {
  const bf16* x; long ldx;
  const bf16* w;            // [rows, K], K contiguous; rows = N (plain) or 2N (swiglu: gate rows then up rows)
  const bf16* norm_w; float eps; int zero_centered;
  const bf16* residual; long ldr;
  void* y; long ldy; int out_f32;
  int T, N, K, mode;
};

template <int T, int R>
__global__ void __launch_bounds__(256) gemv_kernel(GemvParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* xs = reinterpret_cast<bf16*>(smem_raw);
  __shared__ float red[T * 33];
  grid_dep_launch();
  const int t0 = blockIdx.y * T;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (blockIdx.x * 8 + warp) * R;
  if (p.mode == 0) {
    const bf16* rows[R];
#pragma unroll
    for (int r = 0; r < R; ++r) rows[r] = (n0 + r < p.N) ? p.w + (long)(n0 + r) * p.K : nullptr;
    RowBatch<R> pf;
    prefetch_rows<R>(rows, p.K, pf);
    request_gain(p.norm_w, p.K);
    grid_dep_wait();
    stage_x<T>(xs, p.x, p.ldx, t0, p.T, p.K, p.norm_w, p.eps, p.zero_centered != 0, red);
    if (n0 >= p.N) return;
    float acc[R][T];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int t = 0; t < T; ++t) acc[r][t] = 0.f;
    warp_rows_dot<T, R>(rows, xs, p.K, acc, pf);
    warp_reduce_acc<T, R>(acc);
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (n0 + r >= p.N) continue;
#pragma unroll
        for (int t = 0; t < T; ++t) {
          if (t0 + t >= p.T) continue;
          float v = acc[r][t];
          if (p.residual) v = bf16_round(v) + __bfloat162float(p.residual[(long)(t0 + t) * p.ldr + n0 + r]);
          if (p.out_f32) reinterpret_cast<float*>(p.y)[(long)(t0 + t) * p.ldy + n0 + r] = v;
          else reinterpret_cast<bf16*>(p.y)[(long)(t0 + t) * p.ldy + n0 + r] = __float2bfloat16_rn(v);
        }
      }
    }
  } else {
    // swiglu: output feature j uses gate row j and up row N + j
    const bf16* rows[2 * R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool ok = n0 + r < p.N;
      rows[r] = ok ? p.w + (long)(n0 + r) * p.K : nullptr;
      rows[R + r] = ok ? p.w + (long)(p.N + n0 + r) * p.K : nullptr;
    }
    RowBatch<2 * R> pf;
    prefetch_rows<2 * R>(rows, p.K, pf);
    request_gain(p.norm_w, p.K);
    grid_dep_wait();
    stage_x<T>(xs, p.x, p.ldx, t0, p.T, p.K, p.norm_w, p.eps, p.zero_centered != 0, red);
    if (n0 >= p.N) return;
    float acc[2 * R][T];
#pragma unroll
    for (int r = 0; r < 2 * R; ++r)
#pragma unroll
      for (int t = 0; t < T; ++t) acc[r][t] = 0.f;
    warp_rows_dot<T, 2 * R>(rows, xs, p.K, acc, pf);
    warp_reduce_acc<T, 2 * R>(acc);
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (n0 + r >= p.N) continue;
#pragma unroll
        for (int t = 0; t < T; ++t) {
          if (t0 + t >= p.T) continue;
          const float g = bf16_round(acc[r][t]), u = bf16_round(acc[R + r][t]);
          reinterpret_cast<bf16*>(p.y)[(long)(t0 + t) * p.ldy + n0 + r] = __float2bfloat16_rn(silu(g) * u);
        }
      }
    }
  }
}

template <int T, int R>
int launch_gemv(const GemvParams& p, cudaStream_t s) {
  const size_t smem = (size_t)T * p.K * sizeof(bf16);
  auto k = gemv_kernel<T, R>;
  if (int rc = opt_in_smem(k, smem)) return rc;
  dim3 grid((p.N + 8 * R - 1) / (8 * R), (p.T + T - 1) / T);
  return launch_chain(k, grid, dim3(256), smem, s, p);
}

// Rows (or pairs of them) of the matrix to a warp.
//   one row of x        the fewest that leave no more CTAs than run at once, two on an SM (a second wave of a quarter of the CTAs costs as much as the first). Many
//                       columns that take several waves anyway: four rows, whose loads are in flight together. K 2048, us: N 3072 6.4 by one, 4.1 by two;
//                       N 8192 13.2, 9.2 by two, 6.9 by four; gated 6144 11.4 by two pairs, 9.7 by three
//   two to eight        a row's operands in registers serve more products, so that three and four are better as soon as one does not fill the chip: whichever has
//                       the least to do in its waves, of which eight rows get one CTA an SM (registers). K 2048, us by one, two, three, four: two rows N 3072 8.4,
//                       7.5, 6.1, 6.0, N 6144 12.6, 11.2, 7.1, 11.4; four rows N 6144 25.1, 17.4, 11.3, 18.3, N 8192 32.5, 19.7, 19.4, 18.8; eight rows N 3072
//                       28.1, 24.2, 13.6, 16.1, N 4096 31.8, 24.4, 26.4, 16.5. Pairs, by one, two, three: two rows N 3072 9.4, 12.5, 10.1, N 12288 27.6, 32.3, 22.9; four rows N 8192 35.2, 26.4, 29.2; eight rows N 3072 30.0, 30.5, 20.1
template <int T>
int dispatch_rows(const GemvParams& p, cudaStream_t s) {
  if (p.N <= 296 * 8) return launch_gemv<T, 1>(p, s);
  if constexpr (T == 1) {
    if (p.mode) {
      if (p.N <= 296 * 16 || p.N > 296 * 24) return launch_gemv<T, 2>(p, s);
      return launch_gemv<T, 3>(p, s);
    }
    if (p.N <= 296 * 16) return launch_gemv<T, 2>(p, s);
    return launch_gemv<T, 4>(p, s);
  } else {
    auto waves_of = [&](int r) { return ((p.N + 8 * r - 1) / (8 * r) + (T == 8 ? 147 : 295)) / (T == 8 ? 148 : 296) * r; };
    if (p.mode) {
      if (T == 2) return p.N <= 296 * 16 ? launch_gemv<T, 1>(p, s) : launch_gemv<T, 3>(p, s);
      return waves_of(2) < waves_of(3) ? launch_gemv<T, 2>(p, s) : launch_gemv<T, 3>(p, s);
    }
    if (T < 8 && p.N <= 296 * 16) return launch_gemv<T, 4>(p, s);
    return waves_of(3) < waves_of(4) ? launch_gemv<T, 3>(p, s) : launch_gemv<T, 4>(p, s);
  }
}

// Shared memory of the two kinds: two CTAs with a norm never fit an SM together, nor three of any, but one with and one without do. A layer's linears alternate between
// the kinds, so every SM has one CTA of each of two kernels; where two CTAs of a kernel fit, an SM that became free early took two and another one none (2B
// layer 36 us).
constexpr int SMEM_NORM = 126976, SMEM_PLAIN = 102912;
template <int MR, bool GATED, bool NORM>
using RowsStream = RowStream<MR, NORM ? (MR == 8 ? 10 : 12) : 8, NORM ? (MR == 8 ? 4 : 6) : (MR == 8 ? 3 : 5), MR == 8 ? 33792 : NORM ? 18432 : 13312, GATED ? Rows::GATED : Rows::PLAIN>;

// grid (a CTA for each SM, tiles of MR rows of x)
template <int MR, bool GATED, bool NORM>
__global__ void __launch_bounds__(RS_WARPS * 32, 2) rows_kernel(GemvParams p) {
  using S = RowsStream<MR, GATED, NORM>;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ float sums[RS_WARPS * 8];
  grid_dep_launch();
  const int t0 = blockIdx.y * MR, T = min(MR, p.T - t0);
  S stream;
  stream.start(RowShare{p.w, p.N, p.K, (int)((long)p.N * blockIdx.x / gridDim.x), (int)((long)p.N * (blockIdx.x + 1) / gridDim.x), 0}, smem);
  BfRows<MR, NORM> x{p.x + (long)t0 * p.ldx, p.ldx, p.norm_w, p.eps, p.zero_centered, T};
  x.early(stream);
  grid_dep_wait();
  float first_res = 0.f;          // requested here: behind the sums it was one more trip to L2
  int ft, fn;
  if (!GATED && p.residual && stream.first_result(T, &ft, &fn)) first_res = __bfloat162float(p.residual[(long)(t0 + ft) * p.ldr + fn]);
  x.prepare(stream, sums);
  auto out = [&](int t, int n, float v, float u, bool first) {
    if (GATED) {
      const float g = bf16_round(v);
      reinterpret_cast<bf16*>(p.y)[(long)(t0 + t) * p.ldy + n] = __float2bfloat16_rn(silu(g) * bf16_round(u));
      return;
    }
    if (p.residual) v = bf16_round(v) + (first ? first_res : __bfloat162float(p.residual[(long)(t0 + t) * p.ldr + n]));
    if (p.out_f32) reinterpret_cast<float*>(p.y)[(long)(t0 + t) * p.ldy + n] = v;
    else reinterpret_cast<bf16*>(p.y)[(long)(t0 + t) * p.ldy + n] = __float2bfloat16_rn(v);
  };
  stream.run(x, T, out);
}

template <int MR, bool GATED, bool NORM>
int launch_rows(const GemvParams& p, cudaStream_t s) {
  constexpr int smem = NORM ? SMEM_NORM : SMEM_PLAIN;
  static_assert(RowsStream<MR, GATED, NORM>::SMEM <= smem, "ring, sums and rows");
  auto k = rows_kernel<MR, GATED, NORM>;
  if (int rc = opt_in_smem(k, smem)) return rc;
  if (int rc = (int)cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared)) return rc;
  return launch_chain(k, dim3(tc::device_sms(), (p.T + MR - 1) / MR), dim3(RS_WARPS * 32), (size_t)smem, s, p);
}
template <int MR>
int dispatch_rows_stream(const GemvParams& p, cudaStream_t s) {
  if (p.mode) return p.norm_w ? launch_rows<MR, true, true>(p, s) : launch_rows<MR, true, false>(p, s);
  return p.norm_w ? launch_rows<MR, false, true>(p, s) : launch_rows<MR, false, false>(p, s);
}

// The projection of a grouped-query layer with what comes behind it: rows of q and k are turned, keys and values go to their pages. A result is the pair of columns that a
// rotation mixes, so no other launch has to wait for the row: 2B model, a step of one row 4.4 us a layer for the kernel that did it (decode_gqa.cu), of eight rows 3.9.
// q lands in `y`; angles, roundings and pages are that kernel's.
struct QkvParams {
  GemvParams g;
  const int32_t *positions, *slots, *page_table;
  int max_pages, page_tokens, num_pages;
  bf16 *k_cache, *v_cache;
  int Hq, Hkv, half;
  float theta;
  uint32_t* status;
};
template <int MR>
__global__ void __launch_bounds__(RS_WARPS * 32, 2) qkv_rows_kernel(QkvParams q) {
  using S = RowStream<MR, MR == 8 ? 10 : 12, MR == 8 ? 4 : 6, MR == 8 ? 33792 : 18432, Rows::PAIRS>;
  const GemvParams& p = q.g;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ float sums[RS_WARPS * 8];
  grid_dep_launch();
  S stream;
  stream.start(RowShare{p.w, p.N, p.K, (int)((long)p.N * blockIdx.x / gridDim.x), (int)((long)p.N * (blockIdx.x + 1) / gridDim.x), q.half}, smem);
  BfRows<MR, true> x{p.x, p.ldx, p.norm_w, p.eps, p.zero_centered, p.T};
  x.early(stream);
  grid_dep_wait();
  // where row t's keys and values go (-1: nowhere), whether the head turns (values and rows that are not there do not), and the angle of pair j
  struct Place {
    long row;
    bool turns;
    float c, s;
  };
  auto place = [&](int t, int n) {
    Place at{-1, false, 1.f, 0.f};
    const int pos = q.positions[t], h = n / q.half, j = n - h * q.half;
    if (pos < 0) return at;
    if (h >= q.Hq) {
      const int lp = pos / q.page_tokens, page = lp < q.max_pages ? q.page_table[(long)q.slots[t] * q.max_pages + lp] : -1;
      if (page >= 0 && page < q.num_pages) at.row = (long)page * q.page_tokens + pos % q.page_tokens;
      else if (q.status) atomicOr(q.status, IFAB_STATUS_BAD_INDEX);
    }
    if (h < q.Hq + q.Hkv) {
      at.turns = true;
      const float inv_freq = exp2f(-(2.f * (float)j / (float)(2 * q.half)) * log2f(q.theta));
      sincosf((float)pos * inv_freq, &at.s, &at.c);
      at.c = bf16_round(at.c);
      at.s = bf16_round(at.s);
    }
    return at;
  };
  Place mine{-1, false, 1.f, 0.f};       // requested here: behind the sums it was two more trips to L2
  int ft, fn;
  if (stream.first_result(p.T, &ft, &fn)) mine = place(ft, fn);
  x.prepare(stream, sums);
  auto out = [&](int t, int n, float v, float u, bool first) {
    const Place at = first ? mine : place(t, n);
    const int h = n / q.half, j = n - h * q.half, hd = 2 * q.half;
    bf16 lo = __float2bfloat16_rn(v), hi = __float2bfloat16_rn(u);
    if (at.turns) {          // others are copied: by cosine 1 and sine 0 an infinite column would make NaN of its partner
      const float a = __bfloat162float(lo), b = __bfloat162float(hi);
      lo = __float2bfloat16_rn(a * at.c - b * at.s);
      hi = __float2bfloat16_rn(b * at.c + a * at.s);
    }
    bf16* to = reinterpret_cast<bf16*>(p.y) + (long)t * p.ldy + h * hd + j;
    if (h >= q.Hq) {
      if (at.row < 0) return;
      const bool key = h < q.Hq + q.Hkv;
      to = (key ? q.k_cache : q.v_cache) + (at.row * q.Hkv + (h - q.Hq - (key ? 0 : q.Hkv))) * hd + j;
    }
    to[0] = lo;
    to[q.half] = hi;
  };
  stream.run(x, p.T, out);
}
template <int MR>
int launch_qkv(const QkvParams& q, cudaStream_t s) {
  auto k = qkv_rows_kernel<MR>;
  if (int rc = opt_in_smem(k, SMEM_NORM)) return rc;
  if (int rc = (int)cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared)) return rc;
  return launch_chain(k, dim3(tc::device_sms()), dim3(RS_WARPS * 32), (size_t)SMEM_NORM, s, q);
}

// ----------------------------------------------------------------------------------------------
// Row-parallel linear + one-shot all-reduce (protocol in oneshot_ar.cuh).
// Every CTA owns a slab of 8*R output columns for all T tokens; only same-index CTAs of the ranks
// synchronise, so the transfer of early slabs overlaps the math of late ones.
// ----------------------------------------------------------------------------------------------
struct ArParams {
  GemvParams g;
  FabricView fv;
  uint64_t* seq;         // local call counter (read by all CTAs, advanced by the last one)
  uint32_t* done;        // local ticket counter
  float* y_f32;          // optional f32 copy of the reduced output [T, N]
};

template <int T, int R>
__global__ void __launch_bounds__(256) gemv_allreduce_kernel(ArParams a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const GemvParams& p = a.g;
  bf16* xs = reinterpret_cast<bf16*>(smem_raw);
  __shared__ float red[T * 33];
  __shared__ float slab[T * 8 * R];
  __shared__ int timed_out;
  grid_dep_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int RPC = 8 * R;
  const int nbase = blockIdx.x * RPC;
  const int n0 = nbase + warp * R;
  const bf16* rows[R];
#pragma unroll
  for (int r = 0; r < R; ++r) rows[r] = (n0 + r < p.N) ? p.w + (long)(n0 + r) * p.K : nullptr;
  RowBatch<R> pf;
  prefetch_rows<R>(rows, p.K, pf);
  grid_dep_wait();
  if (threadIdx.x == 0) timed_out = 0;
  stage_x<T>(xs, p.x, p.ldx, 0, p.T, p.K, p.norm_w, p.eps, p.zero_centered != 0, red);
  {
    float acc[R][T];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int t = 0; t < T; ++t) acc[r][t] = 0.f;
    warp_rows_dot<T, R>(rows, xs, p.K, acc, pf);
    warp_reduce_acc<T, R>(acc);
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int t = 0; t < T; ++t) slab[t * RPC + warp * R + r] = acc[r][t];
    }
  }
  __syncthreads();
  oneshot_allreduce_slab<T, RPC>(slab, a.fv, a.seq, a.done, nbase, p.T, p.N, p.residual, p.ldr,
                                 reinterpret_cast<bf16*>(p.y), p.ldy, a.y_f32, &timed_out);
}

template <int T, int R>
int launch_ar(const ArParams& a, cudaStream_t s) {
  const size_t smem = (size_t)T * a.g.K * sizeof(bf16);
  auto k = gemv_allreduce_kernel<T, R>;
  if (int rc = opt_in_smem(k, smem)) return rc;
  dim3 grid((a.g.N + 8 * R - 1) / (8 * R));
  return launch_chain(k, grid, dim3(256), smem, s, a);
}

template <int T>
int dispatch_ar(const ArParams& a, cudaStream_t s) {
  // keep the grid <= 296 CTAs (two per SM) so every CTA of every rank is co-resident: CTAs with the
  // same index wait on one another across GPUs.
  const int n = a.g.N;
  if ((n + 7) / 8 <= 296) return launch_ar<T, 1>(a, s);
  if ((n + 15) / 16 <= 296) return launch_ar<T, 2>(a, s);
  if ((n + 31) / 32 <= 296) return launch_ar<T, 4>(a, s);
  return -2;
}

}  // namespace

extern "C" int ifab_gemv_bf16(const void* x, long ldx, const void* w, const void* norm_w, float eps, int zero_centered,
                              const void* residual, long ldr, void* y, long ldy, int out_f32, int T, int N, int K,
                              int mode, void* stream) {
  if (K % 8 != 0 || ldx % 8 != 0) return -1;
  GemvParams p{(const bf16*)x, ldx, (const bf16*)w, (const bf16*)norm_w, eps, zero_centered,
               (const bf16*)residual, ldr, y, ldy, out_f32, T, N, K, mode};
  cudaStream_t s = (cudaStream_t)stream;
  if (T <= 1) return dispatch_rows<1>(p, s);
  if (T <= 2) return dispatch_rows<2>(p, s);
  if (T <= 4) return dispatch_rows<4>(p, s);
  return dispatch_rows<8>(p, s);
}

// The same by rings in shared memory (row_stream.cuh), for chains of kernels that leave L1 alone: a ring wants most of an SM's memory as shared memory, and kernels that
// keep 128 KB of loads in flight in registers (the experts' and the form above) lose a quarter of their rate beside it. x, w and norm_w on 16 bytes.
extern "C" int ifab_gemv_rows_bf16(const void* x, long ldx, const void* w, const void* norm_w, float eps, int zero_centered, const void* residual, long ldr, void* y,
                                   long ldy, int out_f32, int T, int N, int K, int mode, void* stream) {
  const uintptr_t bits = (uintptr_t)x | (uintptr_t)w | (uintptr_t)norm_w;
  if (T < 1 || N < 1 || K < 8 || K % 8 != 0 || ldx % 8 != 0 || bits % 16 != 0 || mode < 0 || mode > 1 || (mode && (residual || out_f32))) return -1;
  GemvParams p{(const bf16*)x, ldx, (const bf16*)w, (const bf16*)norm_w, eps, zero_centered, (const bf16*)residual, ldr, y, ldy, out_f32, T, N, K, mode};
  return T <= 2 ? dispatch_rows_stream<2>(p, (cudaStream_t)stream) : dispatch_rows_stream<8>(p, (cudaStream_t)stream);
}

// q [T, Hq * head_dim] (into y), keys and values (into their pages) of norm(x) w^T with w = [q heads | k heads | v heads] rows; all columns of a head of q and k turn.
// One to eight rows; a row at position -1 writes its q only.
extern "C" int ifab_qkv_rows_bf16(const void* x, long ldx, const void* w, const void* norm_w, float eps, void* y, long ldy, const int32_t* positions,
                                  const int32_t* slots, const int32_t* page_table, int max_pages, int page_tokens, void* k_cache, void* v_cache, int num_pages, int T,
                                  int Hq, int Hkv, int head_dim, int K, float theta, uint32_t* status, void* stream) {
  const uintptr_t bits = (uintptr_t)x | (uintptr_t)w | (uintptr_t)norm_w;
  if (T < 1 || T > 8 || K < 8 || K % 8 != 0 || ldx % 8 != 0 || bits % 16 != 0 || !norm_w || head_dim < 2 || head_dim % 2 || Hq < 1 || Hkv < 1 || page_tokens < 1) return -1;
  QkvParams q{{(const bf16*)x, ldx, (const bf16*)w, (const bf16*)norm_w, eps, 0, nullptr, 0, y, ldy, 0, T, (Hq + 2 * Hkv) * (head_dim / 2), K, 0},
              positions, slots, page_table, max_pages, page_tokens, num_pages, (bf16*)k_cache, (bf16*)v_cache, Hq, Hkv, head_dim / 2, theta, status};
  return T <= 2 ? launch_qkv<2>(q, (cudaStream_t)stream) : launch_qkv<8>(q, (cudaStream_t)stream);
}

extern "C" int ifab_gemv_allreduce_bf16(const void* x, long ldx, const void* w, const void* residual, long ldr,
                                        void* y, long ldy, void* y_f32, int T, int N, int K,
                                        const IfabFabric* fab, void* stream) {
  if (K % 8 != 0 || ldx % 8 != 0 || T > 8 || T < 1) return -1;
  ArParams a;
  a.g = GemvParams{(const bf16*)x, ldx, (const bf16*)w, nullptr, 0.f, 0, (const bf16*)residual, ldr, y, ldy, 0, T, N, K, 0};
  if (int rc = fabric_view(fab, &a.fv)) return rc;
  a.seq = fab->seq;
  a.done = fab->done;
  a.y_f32 = (float*)y_f32;
  if ((size_t)fab->world * T * N * sizeof(uint64_t) > fab->ll_half_bytes) return -3;
  if ((size_t)fab->world * 296 > fab->flag_half_words) return -4;
  cudaStream_t s = (cudaStream_t)stream;
  if (T <= 1) return dispatch_ar<1>(a, s);
  if (T <= 2) return dispatch_ar<2>(a, s);
  if (T <= 4) return dispatch_ar<4>(a, s);
  return dispatch_ar<8>(a, s);
}
