// Decode-time expert FFN over block-scaled fp8 (e4m3) expert weights.
//
// Storage: a weight matrix [rows, K] is kept as one byte per element plus one f32 scale per 1 x 128 block of a row
// (scales[row][ceil(K / 128)]); the represented value is fp8(w[row][k]) * scale[row][k / 128]. Decode linears are bound
// by the HBM stream of the weights, so halving the bytes of the expert matrices - 3/4 of the bytes a token touches in a
// mixture-of-experts layer - is what this buys. Two forms:
//   expert_gate_up_kernel, expert_down_kernel (one rank)   every listed expert is streamed through rings in shared memory once for all
//                       tokens that chose it, its weights widened once, and multiplied on the tensor cores
//   the kernels that mirror the bf16 ones of decode_moe.cu (same grids, same routing inputs, same fused all-reduce)   token by token: gate / up
//                       where the caller says so (small experts, from four ranks on), for more than 1024 experts a rank and where a row doesn't fit
//                       beside the rings; down on several ranks. Every lane converts its 16-byte chunk (16 weights), forms the
//                       chunk's dot product with the activations staged in shared memory, and scales it once
// Reference: W8A8 expert matrices of the 92B program (dequantising grouped matmul, native/src/token_executor.h:640-700).
#include <cuda_fp8.h>

#include <algorithm>

#include "expert_stream.cuh"
#include "gemv.cuh"
#include "ifab_kernels.h"
#include "oneshot_ar.cuh"
#include "row_stream.cuh"

using namespace ifab;

namespace {

constexpr int QBLOCK = 128;
constexpr int MAX_TOPK8 = 16;

// Dot product of one 16-byte chunk (16 fp8 weights) with 16 activations held as f16: the weights convert pairwise to f16
// (one instruction per pair) and multiply-accumulate as half2, eight terms per half, before ONE conversion to f32 - three
// times fewer instructions than converting every weight to f32, which is what makes the halved bytes show up as time.
// The activations are staged scaled by kXScale so that eight products of a weight (|w| <= 448 after block scaling) and an
// activation stay far inside the f16 range; the caller multiplies the result by 1 / kXScale together with the block scale.
constexpr float kXScale = 1.f / 16.f;
__device__ __forceinline__ float dot16_e4m3_f16(const uint4& w, const __half2* xh) {
  const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
  __half2 acc = __float2half2_rn(0.f);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)((ww[i] >> (16 * h)) & 0xffffu), __NV_E4M3);
      acc = __hfma2(*reinterpret_cast<const __half2*>(&hr), xh[i * 2 + h], acc);
    }
  }
  const float2 f = __half22float2(acc);
  return f.x + f.y;
}
// 8 bf16 -> 8 f16 scaled by kXScale
__device__ __forceinline__ uint4 bf16x8_to_scaled_f16(const uint4& v) {
  float f[8];
  unpack8(v, f);
  uint4 o;
  __half2* h = reinterpret_cast<__half2*>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i] * kXScale, f[2 * i + 1] * kXScale);
  return o;
}

// ---- quantiser: one warp per (row, block) ------------------------------------------------------------
__global__ void __launch_bounds__(256) quantize_fp8_block_kernel(const bf16* __restrict__ w, long ldw, long rows, int K, uint8_t* q,
                                                                 float* scales) {
  const int nb = (K + QBLOCK - 1) / QBLOCK;
  const long item = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (item >= rows * nb) return;
  const long row = item / nb;
  const int b = (int)(item % nb), lane = threadIdx.x & 31;
  float v[4];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = b * QBLOCK + lane * 4 + i;
    v[i] = k < K ? __bfloat162float(w[row * ldw + k]) : 0.f;
    amax = fmaxf(amax, fabsf(v[i]));
  }
  amax = warp_max(amax);
  const float scale = amax > 0.f ? __fdiv_rn(amax, 448.f) : 1.f;
  if (lane == 0) scales[row * nb + b] = scale;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = b * QBLOCK + lane * 4 + i;
    if (k < K) q[row * (long)K + k] = (uint8_t)__nv_cvt_float_to_fp8(__fdiv_rn(v[i], scale), __NV_SATFINITE, __NV_E4M3);
  }
}

// ---- dequantiser: 16 values per thread (one 16-byte load, two 16-byte stores); K % 16 == 0 ------------------------------------------
// out = bf16(fp8(q) * scale): the operand form of the tensor-core prompt path, which widens one layer's experts at a time
__global__ void __launch_bounds__(256) dequantize_fp8_block_kernel(const uint8_t* __restrict__ q, const float* __restrict__ scales, long rows, int K,
                                                                   bf16* __restrict__ out) {
  grid_dep_launch();
  grid_dep_wait();
  const int per_row = K / 16, nb = (K + QBLOCK - 1) / QBLOCK;
  const long total = rows * per_row;
  for (long item = (long)blockIdx.x * blockDim.x + threadIdx.x; item < total; item += (long)gridDim.x * blockDim.x) {
    const long row = item / per_row;
    const int c = (int)(item % per_row) * 16;
    const uint4 raw = __ldcs(reinterpret_cast<const uint4*>(q + row * (long)K + c));
    const float sc = scales[row * nb + c / QBLOCK];
    const uint8_t* b = reinterpret_cast<const uint8_t*>(&raw);
    float f[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) f[i] = __half2float(__half(__nv_cvt_fp8_to_halfraw(b[i], __NV_E4M3))) * sc;
    uint4* dst = reinterpret_cast<uint4*>(out + row * (long)K + c);
    dst[0] = pack8(f);
    dst[1] = pack8(f + 8);
  }
}

// ---- gate/up -------------------------------------------------------------------------------------------
struct GateUp8Params {
  const bf16* x; long ldx; const bf16* norm_w; float eps;
  const int32_t* ids; int T, D, F, topk, e0, e_local;
  const uint8_t* w_gu; const float* s_gu; const uint8_t* w_sgu; const float* s_sgu; int Fs;
  bf16* act;
};

// grid: (ceil(F/16), T*topk + T), the layout of the bf16 kernel: a warp owns gate rows j0, j0+1 and up rows j0, j0+1.
__global__ void __launch_bounds__(256) moe_gate_up_fp8_kernel(GateUp8Params p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* xs = reinterpret_cast<bf16*>(smem_raw);
  __shared__ float red[33];
  grid_dep_launch();
  const int routes = p.T * p.topk;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j0 = (blockIdx.x * 8 + warp) * 2;
  const bool shared_col = (int)blockIdx.y >= routes;
  const int nb = (p.D + QBLOCK - 1) / QBLOCK, chunks = p.D >> 4;
  const uint8_t* rows[4] = {nullptr, nullptr, nullptr, nullptr};
  const float* srow[4] = {nullptr, nullptr, nullptr, nullptr};
  int t, slot, Fcur;
  const uint8_t* W;
  const float* S;
  if (shared_col) {
    t = blockIdx.y - routes;
    slot = p.topk;
    W = p.w_sgu;
    S = p.s_sgu;
    Fcur = W ? p.Fs : 0;
  } else {
    grid_dep_wait();
    t = blockIdx.y / p.topk;
    slot = blockIdx.y % p.topk;
    const int e = p.ids[blockIdx.y];
    if (e < p.e0 || e >= p.e0 + p.e_local) return;
    W = p.w_gu + (size_t)(e - p.e0) * 2 * p.F * p.D;
    S = p.s_gu + (size_t)(e - p.e0) * 2 * p.F * nb;
    Fcur = p.F;
  }
  if (j0 < Fcur) {
    const int r[4] = {j0, j0 + 1, Fcur + j0, Fcur + j0 + 1};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if ((i & 1) && j0 + 1 >= Fcur) continue;
      rows[i] = W + (size_t)r[i] * p.D;
      srow[i] = S + (size_t)r[i] * nb;
    }
  }
  constexpr int U = 4;   // 16 chunks of 16 bytes in flight per lane, over 4 rows
  uint4 pf[U][4];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int c = lane + u * 32;
#pragma unroll
    for (int i = 0; i < 4; ++i) pf[u][i] = (c < chunks && rows[i]) ? ld_stream16(rows[i] + (size_t)c * 16) : make_uint4(0, 0, 0, 0);
  }
  if (shared_col) grid_dep_wait();
  if ((int)blockIdx.x * 16 >= Fcur) return;
  stage_x<1>(xs, p.x, p.ldx, t, p.T, p.D, p.norm_w, p.eps, false, red);
  // the normalised row, in place, as scaled f16 (same 2 bytes per element)
  for (int c = threadIdx.x; c < (p.D >> 3); c += blockDim.x) {
    uint4* q = reinterpret_cast<uint4*>(xs + c * 8);
    *q = bf16x8_to_scaled_f16(*q);
  }
  __syncthreads();
  const __half2* xh = reinterpret_cast<const __half2*>(xs);
  if (j0 >= Fcur) return;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int c0 = lane; c0 < chunks; c0 += 32 * U) {
    if (c0 != lane) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int c = c0 + u * 32;
#pragma unroll
        for (int i = 0; i < 4; ++i) pf[u][i] = (c < chunks && rows[i]) ? ld_stream16(rows[i] + (size_t)c * 16) : make_uint4(0, 0, 0, 0);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = c0 + u * 32;
      if (c < chunks) {
        __half2 xv[8];
        *reinterpret_cast<uint4*>(xv) = *reinterpret_cast<const uint4*>(xh + c * 8);
        *reinterpret_cast<uint4*>(xv + 4) = *reinterpret_cast<const uint4*>(xh + c * 8 + 4);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (rows[i] == nullptr) continue;
          acc[i] = fmaf(__ldg(srow[i] + (c >> 3)), dot16_e4m3_f16(pf[u][i], xv), acc[i]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] = warp_sum(acc[i]);
  if (lane == 0) {
    constexpr float un = 1.f / kXScale;
    bf16* out = p.act + ((size_t)t * (p.topk + 1) + slot) * p.F;
    out[j0] = __float2bfloat16_rn(silu(bf16_round(acc[0] * un)) * bf16_round(acc[2] * un));
    if (j0 + 1 < Fcur) out[j0 + 1] = __float2bfloat16_rn(silu(bf16_round(acc[1] * un)) * bf16_round(acc[3] * un));
  }
}

// ---- both halves with every expert read once -----------------------------------------------------------
// A step's tokens choose overlapping experts, and converting a weight costs more than multiplying it: here an expert's weights are read and converted once, for all of its
// tokens, and multiplied on the tensor cores (m16n8k16 in f16, f32 sums: sixteen rows of weights against eight tokens). A CTA an SM streams its share through rings
// like those of row_stream.cuh, sixteen rows by 256 columns (gate / up) or 32 rows by 128 (down) a warp and stage, block scales beside them; a product of a block of
// 128 columns is scaled once. The shared expert comes first: its weights are on the way before the wait for the router.
// Bound by the bytes of the chosen experts. 8 tokens of 8 among 96 experts and a shared one, 4096 x 1536: a token at a time on the CUDA cores
// gate / up 212 us and down 101, so 108 (642 MB: 5.9 TB/s) and 78 (321 MB: 4.1 TB/s, half of its instructions being conversions).
__device__ __forceinline__ void mma16816_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// four fp8 values as two pairs of f16
__device__ __forceinline__ uint2 halves_of(uint32_t w) {
  const __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)w, __NV_E4M3), hi = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w >> 16), __NV_E4M3);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}
// sixteen columns of sixteen rows (lane: rows g and g + 8) against eight tokens: x, x + 1 hold the lane's token's values of them
__device__ __forceinline__ void mma_piece(float (&d)[4], const uint4& w, const uint4& w8, const uint4& x, const uint4& x1) {
  const uint2 a = halves_of(w.x), a8 = halves_of(w8.x), b = halves_of(w.y), b8 = halves_of(w8.y), c = halves_of(w.z), c8 = halves_of(w8.z), e = halves_of(w.w), e8 = halves_of(w8.w);
  mma16816_f16(d, a.x, a8.x, a.y, a8.y, x.x, x.y);
  mma16816_f16(d, b.x, b8.x, b.y, b8.y, x.z, x.w);
  mma16816_f16(d, c.x, c8.x, c.y, c8.y, x1.x, x1.y);
  mma16816_f16(d, e.x, e8.x, e.y, e8.y, x1.z, x1.w);
}
__device__ __forceinline__ void copy4(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live ? 4 : 0) : "memory");
}
// where piece c (16 bytes) of row r lies within 128 bytes: a quarter of a warp writes a row and reads half of two, in either case without meeting a bank twice
__device__ __forceinline__ int swizzled(int c, int r) { return c ^ ((r & 1) << 2 | (r >> 1 & 3)); }

constexpr int XP_STAGE = 4096, XP_SCALES = 128, XP_DEPTH = 3, XP_TILES = 4;
constexpr int XP_RING = 8 * XP_DEPTH * (XP_STAGE + XP_SCALES), XP_RED = 8 * XP_TILES * 128 * 4;

// A CTA's share of gate / up: first pairs of the shared expert, then eights of pairs of the listed experts
__global__ void __launch_bounds__(256, 1) expert_gate_up_kernel(GateUp8Params p) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ RouteList list;
  __shared__ float sums[RS_WARPS * 8];
  __shared__ int tile_entry[XP_TILES], tile_row[XP_TILES], tile_live[XP_TILES];
  grid_dep_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, nb = (p.D + QBLOCK - 1) / QBLOCK, chunks = (p.D + 2047) / 2048;
  const uint32_t ring = smem_addr(smem) + warp * XP_DEPTH * (XP_STAGE + XP_SCALES);
  float* red = reinterpret_cast<float*>(smem + XP_RING);
  struct {
    struct { int K; } s;
    uint32_t xs;
    int pitch, warp, lane;
    __device__ bool fits(int) const { return true; }
  } rows{{p.D}, smem_addr(smem) + XP_RING + XP_RED, (p.D * 2 + 127) / 128 * 128 + 16, warp, lane};
  const int lo = p.w_sgu ? (int)((long)p.Fs * blockIdx.x / gridDim.x) : 0, hi = p.w_sgu ? (int)((long)p.Fs * (blockIdx.x + 1) / gridDim.x) : 0, shared_tiles = (hi - lo + 7) / 8;
  const int eights = p.F / 8;
  int tiles = shared_tiles, first = 0;         // of this CTA; first eight of the listed experts'
  // the tile a cursor stands on: entry (-1: the shared expert), first pair, pairs
  struct Cursor {
    int i, entry, row;
  };
  auto begin = [&](Cursor& c) {
    c.i = 0;
    c.entry = shared_tiles ? -1 : first / eights;
    c.row = shared_tiles ? lo : (first - c.entry * eights) * 8;
  };
  auto advance = [&](Cursor& c) {
    if (++c.i == shared_tiles) {
      c.entry = first / eights;
      c.row = (first - c.entry * eights) * 8;
    } else if ((c.row += 8) == p.F && c.entry >= 0) {
      c.row = 0;
      ++c.entry;
    }
  };
  Cursor ask;
  int k_ask = 0, asked = 0;
  auto request = [&](int at) {
    if (ask.i < tiles) {
      const bool shared = ask.entry < 0;
      const int F = shared ? p.Fs : p.F, live = shared ? hi - ask.row : 8;
      const size_t e = shared ? 0 : list.expert[ask.entry];
      const uint8_t* w = (shared ? p.w_sgu : p.w_gu + e * 2 * p.F * p.D) + (size_t)ask.row * p.D;
      const float* sc = (shared ? p.s_sgu : p.s_gu + e * 2 * p.F * nb) + (size_t)ask.row * nb;
      const uint32_t to = ring + at * (XP_STAGE + XP_SCALES);
      const int col = k_ask * 2048 + warp * 256 + (lane & 7) * 16, r0 = lane >> 3;
      const uint32_t at0 = to + r0 * 128 + swizzled(lane & 7, r0) * 16;      // rows r0 and r0 + 4 of the gate rows, the same of the up rows
      const uint8_t* from = w + (size_t)r0 * p.D + col;
      const size_t four = 4 * (size_t)p.D, up = (size_t)F * p.D;
      const bool in0 = col < p.D, in1 = col + 128 < p.D;
      // rows that are not there may hold anything (a row's sums are its own), columns that are not there are zeros
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint8_t* row = from + (i & 1 ? four : 0) + (i >= 2 ? up : 0);
        const uint32_t dst = (i & 1 ? (at0 ^ 32) + 512 : at0) + (i >> 1) * 2048;
        if (r0 + (i & 1) * 4 < live) {
          copy16(dst, in0 ? row : p.w_gu, in0);
          copy16(dst + 1024, in1 ? row + 128 : p.w_gu, in1);
        }
      }
      const int r = lane >> 1, b = k_ask * 16 + warp * 2 + (lane & 1);
      const bool in = (r & 7) < live && b < nb;
      copy4(to + XP_STAGE + lane * 4, in ? sc + (size_t)((r & 7) + (r >= 8 ? F : 0)) * nb + b : p.s_gu, in);
      if (++k_ask == chunks) {
        k_ask = 0;
        advance(ask);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  begin(ask);
  for (; asked < XP_DEPTH && ask.i < shared_tiles; ++asked) request(asked);
  if (p.norm_w) request_gain(p.norm_w, p.D);
  grid_dep_wait();
  // rows of x, normalised on request, as f16 scaled by kXScale
  auto stage = [&](auto x) {
    x.early(rows);
    x.prepare(rows, sums);
  };
  if (p.norm_w) stage(BfRows<8, true>{p.x, p.ldx, p.norm_w, p.eps, 0, p.T});
  else stage(BfRows<8, false>{p.x, p.ldx, nullptr, 0.f, 0, p.T});
  list_routes(list, p.ids, p.T, p.topk, p.e0, p.e_local);
  for (int i = threadIdx.x; i < p.T * (p.D >> 3); i += 256) {
    const int t = i / (p.D >> 3);
    uint4* at = reinterpret_cast<uint4*>(smem + XP_RING + XP_RED + t * rows.pitch) + (i - t * (p.D >> 3));
    *at = bf16x8_to_scaled_f16(*at);
  }
  const long all = (long)list.n * eights;
  first = (int)(all * blockIdx.x / gridDim.x);
  tiles = shared_tiles + (int)(all * (blockIdx.x + 1) / gridDim.x) - first;
  if (ask.i >= shared_tiles) {                 // the cursor was past the shared expert before the list was there
    ask.entry = first / eights;
    ask.row = (first - ask.entry * eights) * 8;
  }
  for (; asked < XP_DEPTH; ++asked) request(asked);
  __syncthreads();
  Cursor use;
  begin(use);
  int slot = 0;
  const bool token = g < p.T;
  const uint32_t xat = rows.xs + g * rows.pitch + warp * 512 + q * 32;
  for (int i0 = 0; i0 < tiles; i0 += XP_TILES) {
    for (int tt = 0; tt < XP_TILES && i0 + tt < tiles; ++tt) {
      if (threadIdx.x == 0) {
        tile_entry[tt] = use.entry;
        tile_row[tt] = use.row;
        tile_live[tt] = use.entry < 0 ? min(8, hi - use.row) : 8;
      }
      advance(use);
      float acc[4] = {0.f, 0.f, 0.f, 0.f};     // gate row g of tokens 2 q and 2 q + 1, up row g of them
#pragma unroll 1
      for (int k = 0; k < chunks; ++k) {
        asm volatile("cp.async.wait_group %0;" ::"n"(XP_DEPTH - 1) : "memory");
        __syncwarp();
        const uint32_t at = ring + slot * (XP_STAGE + XP_SCALES);
        const float2 sg = *reinterpret_cast<const float2*>(smem + (at - smem_addr(smem)) + XP_STAGE + g * 8), su = *reinterpret_cast<const float2*>(smem + (at - smem_addr(smem)) + XP_STAGE + 64 + g * 8);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const uint32_t piece = at + h * 1024 + g * 128 + swizzled(q + 4 * u, g) * 16;
            uint4 x = make_uint4(0, 0, 0, 0), x1 = x;
            if (token && k * 2048 + warp * 256 + h * 128 + (q + 4 * u) * 16 < p.D) {
              const uint32_t from = xat + k * 4096 + h * 256 + u * 128;
              x = ld_shared16(from);
              x1 = ld_shared16(from + 16);
            }
            mma_piece(d, ld_shared16(piece), ld_shared16(piece + 2048), x, x1);
          }
          const float a = h ? sg.y : sg.x, b = h ? su.y : su.x;
          acc[0] = fmaf(a, d[0], acc[0]);
          acc[1] = fmaf(a, d[1], acc[1]);
          acc[2] = fmaf(b, d[2], acc[2]);
          acc[3] = fmaf(b, d[3], acc[3]);
        }
        __syncwarp();                          // the stage is read
        request(slot);
        slot = slot + 1 == XP_DEPTH ? 0 : slot + 1;
      }
      *reinterpret_cast<float4*>(red + ((warp * XP_TILES + tt) * 32 + lane) * 4) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    }
    __syncthreads();
    const int n = min(XP_TILES, tiles - i0);
    for (int i = threadIdx.x; i < n * 64; i += 256) {
      const int tt = i >> 6, r = i & 7, t = i >> 3 & 7, entry = tile_entry[tt];
      if (t >= p.T || r >= tile_live[tt]) continue;
      const int s = entry < 0 ? p.topk : list.slot[entry][t];
      if (s < 0) continue;
      const float* from = red + (tt * 32 + r * 4 + (t >> 1)) * 4 + (t & 1);
      float a = 0.f, b = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        a += from[w * XP_TILES * 128];
        b += from[w * XP_TILES * 128 + 2];
      }
      constexpr float un = 1.f / kXScale;
      p.act[((size_t)t * (p.topk + 1) + s) * p.F + tile_row[tt] + r] = __float2bfloat16_rn(silu(bf16_round(a * un)) * bf16_round(b * un));
    }
    if (i0 + XP_TILES < tiles) __syncthreads();
  }
}

// ---- down + all-reduce ---------------------------------------------------------------------------------
struct Down8Params {
  const bf16* act; const int32_t* ids; const float* wts;
  int T, D, F, topk, e0, e_local;
  const uint8_t* w_down; const float* s_down; const uint8_t* w_sdown; const float* s_sdown; int Fs;
  const bf16* residual; long ldr; bf16* y; long ldy;
  FabricView fv; uint64_t* seq; uint32_t* done;
};

// The K dimension of all local routes of a token is flattened into one space of 16-element chunks, as in the bf16 kernel:
//   y[t][n] = sum_s wgt_s * sum_blocks scale_s[n][b] * dot(W8_s[n, block b], act[t][s][block b])
template <int T, int R>
__global__ void __launch_bounds__(256) moe_down_fp8_allreduce_kernel(Down8Params p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* as = reinterpret_cast<bf16*>(smem_raw);   // [(topk+1)][F] activation rows of the current token, held as scaled f16 (2 bytes each)
  constexpr int RPC = 8 * R;
  constexpr int MAXS = MAX_TOPK8 + 1;
  __shared__ float slab[T * RPC];
  __shared__ int timed_out;
  __shared__ const uint8_t* s_w[MAXS];
  __shared__ const float* s_sc[MAXS];
  __shared__ float s_g[MAXS];
  __shared__ int s_k[MAXS];
  __shared__ int s_cbeg[MAXS + 1];
  __shared__ int s_slot[MAXS];
  __shared__ int s_n;
  grid_dep_launch();
  grid_dep_wait();
  if (gridDim.y > 1) {              // one rank: a CTA per token (T == 1)
    const int t = blockIdx.y;
    p.act += (size_t)t * (p.topk + 1) * p.F;
    p.ids += t * p.topk;
    p.wts += t * p.topk;
    if (p.residual) p.residual += t * p.ldr;
    p.y += t * p.ldy;
    p.T = 1;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nbase = blockIdx.x * RPC, n0 = nbase + warp * R;
  if (threadIdx.x == 0) timed_out = 0;
  for (int t = 0; t < T; ++t) {
    if (t < p.T) {
      __syncthreads();
      if (warp == 0) {
        // route table, one slot per lane (ids and scores of all slots requested at once), compacted with a ballot
        const int slot = lane;
        bool local = false;
        const uint8_t* w = nullptr;
        const float* sc = nullptr;
        float g = 0.f;
        int k = 0;
        if (slot < p.topk) {
          const int e = p.ids[t * p.topk + slot];
          local = e >= p.e0 && e < p.e0 + p.e_local;
          const size_t el = local ? (size_t)(e - p.e0) : 0;
          w = p.w_down + el * p.D * p.F;
          sc = p.s_down + el * p.D * ((p.F + QBLOCK - 1) / QBLOCK);
          g = p.wts[t * p.topk + slot];
          k = p.F;
        } else if (slot == p.topk && p.w_sdown != nullptr) {
          local = true;
          w = p.w_sdown;
          sc = p.s_sdown;
          g = 1.f;
          k = p.Fs;
        }
        const unsigned m = __ballot_sync(0xffffffffu, local);
        const int n = __popc(m & ((1u << lane) - 1u));
        if (local) {
          s_w[n] = w;
          s_sc[n] = sc;
          s_g[n] = g;
          s_k[n] = k;
          s_slot[n] = slot;
          s_cbeg[n] = n * (p.F >> 4);              // every route before the shared expert spans F
        }
        if (lane == 0) {
          const int total_n = __popc(m), shared = (int)((m >> p.topk) & 1u);
          s_cbeg[total_n] = (total_n - shared) * (p.F >> 4) + shared * (p.Fs >> 4);
          s_n = total_n;
        }
      }
      __syncthreads();
      const int n_routes = s_n;
      {
        // activation rows of the local routes -> scaled f16 in shared memory: eight loads in flight per thread
        const int kch0 = max(1, p.F >> 3);
        const int shared_last = (n_routes > 0 && s_slot[n_routes - 1] == p.topk) ? 1 : 0;
        const int total_c = (n_routes - shared_last) * kch0 + shared_last * (p.Fs >> 3);
        constexpr int SB = 8;
        for (int q0 = threadIdx.x; q0 < total_c; q0 += (int)blockDim.x * SB) {
          uint4 v[SB];
          int dst[SB];
#pragma unroll
          for (int j = 0; j < SB; ++j) {
            const int q = q0 + (int)blockDim.x * j;
            dst[j] = -1;
            if (q < total_c) {
              const int i = min(q / kch0, n_routes - 1), c = q - i * kch0;
              v[j] = *reinterpret_cast<const uint4*>(p.act + ((size_t)t * (p.topk + 1) + s_slot[i]) * p.F + c * 8);
              dst[j] = i * p.F + c * 8;
            }
          }
#pragma unroll
          for (int j = 0; j < SB; ++j)
            if (dst[j] >= 0) *reinterpret_cast<uint4*>(as + dst[j]) = bf16x8_to_scaled_f16(v[j]);
        }
      }
      __syncthreads();
      float total[R];
#pragma unroll
      for (int r = 0; r < R; ++r) total[r] = 0.f;
      constexpr int MAXC = 4;   // 16-byte chunks (16 weights) per lane and route held in registers (K <= 2048)
      if ((p.F >> 4) <= 32 * MAXC) {
        // one route at a time, as in the bf16 kernel: base pointers, score and activation row are loop invariants
        for (int i = 0; i < n_routes; ++i) {
          const int k = s_k[i], kch = k >> 4, nbk = (k + QBLOCK - 1) / QBLOCK;
          const uint8_t* wb = s_w[i] + (size_t)n0 * k;
          const float* sb = s_sc[i] + (size_t)n0 * nbk;
          uint4 wv[MAXC][R];
          float sv[MAXC][R];
#pragma unroll
          for (int u = 0; u < MAXC; ++u) {
            const int c = lane + 32 * u;
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const bool in = c < kch && n0 + r < p.D;
              wv[u][r] = in ? ld_stream16(wb + (size_t)r * k + (size_t)c * 16) : make_uint4(0, 0, 0, 0);
              sv[u][r] = in ? __ldg(sb + (size_t)r * nbk + (c >> 3)) : 0.f;
            }
          }
          const float g = s_g[i];
          const bf16* arow_s = as + (size_t)i * p.F;
          float acc[R];
#pragma unroll
          for (int r = 0; r < R; ++r) acc[r] = 0.f;
#pragma unroll
          for (int u = 0; u < MAXC; ++u) {
            const int c = lane + 32 * u;
            if (c < kch) {
              __half2 xv[8];
              const __half2* xa = reinterpret_cast<const __half2*>(arow_s) + c * 8;
              *reinterpret_cast<uint4*>(xv) = *reinterpret_cast<const uint4*>(xa);
              *reinterpret_cast<uint4*>(xv + 4) = *reinterpret_cast<const uint4*>(xa + 4);
#pragma unroll
              for (int r = 0; r < R; ++r) acc[r] = fmaf(sv[u][r], dot16_e4m3_f16(wv[u][r], xv), acc[r]);
            }
          }
#pragma unroll
          for (int r = 0; r < R; ++r) total[r] = fmaf(g * (1.f / kXScale), acc[r], total[r]);
        }
      } else {
      const int chunks = s_cbeg[n_routes];
        const int cpr = p.F >> 4;
        const int n_exp_chunks = (n_routes > 0 && s_slot[n_routes - 1] == p.topk) ? s_cbeg[n_routes - 1] : chunks;
        constexpr int U = 16 / R;
        for (int c0 = lane; c0 < chunks; c0 += 32 * U) {
          uint4 wv[U][R];
          float sv[U][R];
          int route[U], cc[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int c = c0 + u * 32;
            const int i = c < n_exp_chunks ? c / cpr : n_routes - 1;
            route[u] = i;
            cc[u] = c < n_exp_chunks ? c - i * cpr : c - n_exp_chunks;
            if (c < chunks) {
              const int k = s_k[i], nbk = (k + QBLOCK - 1) / QBLOCK;
              const uint8_t* wb = s_w[i] + (size_t)n0 * k + (size_t)cc[u] * 16;
              const float* sb = s_sc[i] + (size_t)n0 * nbk + (cc[u] >> 3);
#pragma unroll
              for (int r = 0; r < R; ++r) {
                const bool in = n0 + r < p.D;
                wv[u][r] = in ? ld_stream16(wb + (size_t)r * k) : make_uint4(0, 0, 0, 0);
                sv[u][r] = in ? __ldg(sb + (size_t)r * nbk) : 0.f;
              }
            } else {
#pragma unroll
              for (int r = 0; r < R; ++r) { wv[u][r] = make_uint4(0, 0, 0, 0); sv[u][r] = 0.f; }
            }
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (c0 + u * 32 < chunks) {
              __half2 xv[8];
              const __half2* xa = reinterpret_cast<const __half2*>(as + (size_t)route[u] * p.F) + cc[u] * 8;
              *reinterpret_cast<uint4*>(xv) = *reinterpret_cast<const uint4*>(xa);
              *reinterpret_cast<uint4*>(xv + 4) = *reinterpret_cast<const uint4*>(xa + 4);
              const float g = s_g[route[u]] * (1.f / kXScale);
#pragma unroll
              for (int r = 0; r < R; ++r) total[r] = fmaf(g * sv[u][r], dot16_e4m3_f16(wv[u][r], xv), total[r]);
            }
          }
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float v = warp_sum(total[r]);
        if (lane == 0) slab[t * RPC + warp * R + r] = v;
      }
    }
  }
  __syncthreads();
  oneshot_allreduce_slab<T, RPC>(slab, p.fv, p.seq, p.done, nbase, p.T, p.D, p.residual, p.ldr, p.y, p.ldy, nullptr, &timed_out);
}

// `tokens` > 1 (one rank, T == 1): a CTA per token and 8 R columns. Tokens one after the other in a CTA (which the exchange of several ranks asks for)
// wait for one route's weights after the other's: 8 tokens of 9 routes, 4096 x 1536: 201 us, a token each 98 us.
template <int T, int R>
int launch_down8(const Down8Params& p, cudaStream_t s, int tokens = 1) {
  const size_t smem = (size_t)(p.topk + 1) * p.F * sizeof(bf16);
  auto k = moe_down_fp8_allreduce_kernel<T, R>;
  if (int rc = opt_in_smem(k, smem)) return rc;
  dim3 grid((p.D + 8 * R - 1) / (8 * R), tokens);
  return launch_chain(k, grid, dim3(256), smem, s, p);
}
template <int T>
int dispatch_down8(const Down8Params& p, cudaStream_t s) {
  if ((p.D + 7) / 8 <= 296) return launch_down8<T, 1>(p, s);
  if ((p.D + 15) / 16 <= 296) return launch_down8<T, 2>(p, s);
  if ((p.D + 31) / 32 <= 296) return launch_down8<T, 4>(p, s);
  return -2;
}

// A CTA's rows of the down projection, 32 at a time, over all experts of all tokens; a warp takes every eighth block of 128 columns (which one, an expert's number says, so that
// a token's sums do not depend on its neighbours'). One rank.
__global__ void __launch_bounds__(256, 1) expert_down_kernel(Down8Params p) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ RouteList list;
  __shared__ float weight[RL_ROUTES][RL_TOKENS];
  grid_dep_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int r0 = (int)((long)p.D * blockIdx.x / gridDim.x), r1 = (int)((long)p.D * (blockIdx.x + 1) / gridDim.x);
  const uint32_t ring = smem_addr(smem) + warp * XP_DEPTH * (XP_STAGE + XP_SCALES);
  float* red = reinterpret_cast<float*>(smem + XP_RING);
  const int nb = (p.F + QBLOCK - 1) / QBLOCK, nbs = p.w_sdown ? (p.Fs + QBLOCK - 1) / QBLOCK : 0;
  int n = 0;                                   // entries
  bool known = false;
  // a warp's blocks: of the shared expert (entry -1), then of the listed ones
  struct Cursor {
    int row, entry, block;
  };
  auto settle = [&](Cursor& c) {               // on to the next block that there is (row r1: none)
    for (;;) {
      if (c.entry < 0 ? c.block < nbs : c.entry < n && c.block < nb) return;
      if (++c.entry >= n) {
        if (!known) return;                    // the list is not there yet
        c.entry = -1;
        c.block = warp;
        c.row += 32;
        if (c.row >= r1) return;
        continue;
      }
      c.block = (warp - list.expert[c.entry] * nb) & 7;
    }
  };
  Cursor ask{r0, -1, warp}, use{r0, -1, warp};
  auto request = [&](int at) {
    const uint32_t to = ring + at * (XP_STAGE + XP_SCALES);
    if (ask.row < r1 && (known || ask.entry < 0)) {
      const bool shared = ask.entry < 0;
      const int F = shared ? p.Fs : p.F, blocks = shared ? nbs : nb;
      const size_t e = shared ? 0 : list.expert[ask.entry];
      const uint8_t* w = (shared ? p.w_sdown : p.w_down + e * p.D * p.F) + (size_t)ask.row * F;
      const float* sc = (shared ? p.s_sdown : p.s_down + e * p.D * nb) + (size_t)ask.row * blocks + ask.block;
      const int live = r1 - ask.row, col = ask.block * 128 + (lane & 7) * 16, row0 = lane >> 3;
      const bool in = col < F;
      const uint8_t* from = in ? w + (size_t)row0 * F + col : p.w_down;
      const size_t four = in ? 4 * (size_t)F : 0;
      const uint32_t at0 = to + row0 * 128 + swizzled(lane & 7, row0) * 16;
      // rows that are not there may hold anything (a row's sums are its own), columns that are not there are zeros
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (row0 + i * 4 < live) copy16((i & 1 ? at0 ^ 32 : at0) + i * 512, from, in);
        from += four;
      }
      copy4(to + XP_STAGE + lane * 4, lane < live ? sc + (size_t)lane * blocks : p.s_down, lane < live);
      ask.block += 8;
      settle(ask);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int asked = 0;
  settle(ask);
  for (; asked < XP_DEPTH && ask.entry < 0 && ask.row == r0; ++asked) request(asked);
  grid_dep_wait();
  if (p.seq && blockIdx.x == 0 && threadIdx.x == 0) *p.seq += 1;
  list_routes(list, p.ids, p.T, p.topk, p.e0, p.e_local);
  for (int i = threadIdx.x; i < list.n * RL_TOKENS; i += 256) {
    const int t = i & 7, s = list.slot[i >> 3][t];
    weight[i >> 3][t] = s >= 0 ? p.wts[t * p.topk + s] : 0.f;
  }
  n = list.n;
  known = true;
  if (ask.entry >= 0) {                        // it had left the shared expert
    ask.entry = -1;
    ask.block = nbs;
    settle(ask);
  }
  for (; asked < XP_DEPTH; ++asked) request(asked);
  __syncthreads();
  settle(use);
  // this lane's token's values of a block: pieces q and q + 4
  uint4 raw[4];
  auto load = [&](const Cursor& c) {
    const int s = g >= p.T || c.row >= r1 ? -1 : c.entry < 0 ? p.topk : list.slot[c.entry][g], F = c.entry < 0 ? p.Fs : p.F;
    const bf16* row = p.act + ((size_t)g * (p.topk + 1) + max(s, 0)) * p.F + c.block * 128;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int col = (q + 4 * u) * 16;
      const bool in = s >= 0 && c.block * 128 + col < F;
      raw[2 * u] = raw[2 * u + 1] = make_uint4(0, 0, 0, 0);
      if (in) {
        raw[2 * u] = ld_row16(row + col);
        raw[2 * u + 1] = ld_row16(row + col + 8);
      }
    }
  };
  load(use);
  int slot = 0;
  for (int row = r0; row < r1; row += 32) {
    float acc[2][4] = {};                      // [sixteen rows][row g of tokens 2 q and 2 q + 1, row g + 8 of them]
    while (use.row == row && (use.entry < 0 ? use.block < nbs : use.entry < n)) {
      uint4 x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = bf16x8_to_scaled_f16(raw[i]);
      float c[2];
      bool his[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = 2 * q + i;
        his[i] = t < p.T && (use.entry < 0 || list.slot[use.entry][t] >= 0);
        c[i] = (use.entry < 0 ? 1.f : weight[use.entry][t]) * (1.f / kXScale);
      }
      use.block += 8;
      settle(use);
      load(use);
      asm volatile("cp.async.wait_group %0;" ::"n"(XP_DEPTH - 1) : "memory");
      __syncwarp();
      const uint32_t at = ring + slot * (XP_STAGE + XP_SCALES);
      const float* scales = reinterpret_cast<const float*>(smem + (at - smem_addr(smem)) + XP_STAGE);
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint32_t piece = at + m * 2048 + g * 128 + swizzled(q + 4 * u, g) * 16;
          mma_piece(d, ld_shared16(piece), ld_shared16(piece + 1024), x[2 * u], x[2 * u + 1]);
        }
        const float a = scales[m * 16 + g], b = scales[m * 16 + 8 + g];
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (his[i]) {
            acc[m][i] = fmaf(c[i] * a, d[i], acc[m][i]);
            acc[m][2 + i] = fmaf(c[i] * b, d[2 + i], acc[m][2 + i]);
          }
      }
      __syncwarp();                            // the stage is read
      request(slot);
      slot = slot + 1 == XP_DEPTH ? 0 : slot + 1;
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) *reinterpret_cast<float4*>(red + ((warp * 2 + m) * 32 + lane) * 4) = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
    __syncthreads();
    for (int i = threadIdx.x; i < 32 * RL_TOKENS; i += 256) {
      const int r = i & 31, t = i >> 5;
      if (t >= p.T || row + r >= r1) continue;
      const float* from = red + ((r >> 4) * 32 + (r & 7) * 4 + (t >> 1)) * 4 + (r >> 3 & 1) * 2 + (t & 1);
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) v += from[w * 256];
      if (p.residual) v = bf16_round(v) + __bfloat162float(p.residual[(long)t * p.ldr + row + r]);
      p.y[(long)t * p.ldy + row + r] = __float2bfloat16_rn(v);
    }
    if (row + 32 < r1) __syncthreads();
  }
}
int launch_expert_down(const Down8Params& p, cudaStream_t s) {
  constexpr int smem = XP_RING + 8 * 2 * 128 * 4;
  if (int rc = opt_in_smem(expert_down_kernel, smem)) return rc;
  if (int rc = (int)cudaFuncSetAttribute(expert_down_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared)) return rc;
  return launch_chain(expert_down_kernel, dim3(tc::device_sms()), dim3(256), (size_t)smem, s, p);
}

}  // namespace

// w: bf16 [rows, K] (row stride ldw); q: u8 [rows, K]; scales: f32 [rows, ceil(K / 128)]
extern "C" int ifab_quantize_fp8_block(const void* w, long ldw, long rows, int K, void* q, float* scales, void* stream) {
  if (rows < 1 || K < 1) return -1;
  const long items = rows * ((K + QBLOCK - 1) / QBLOCK);
  quantize_fp8_block_kernel<<<(unsigned)((items + 7) / 8), 256, 0, (cudaStream_t)stream>>>((const bf16*)w, ldw, rows, K, (uint8_t*)q, scales);
  return (int)cudaGetLastError();
}

// q: u8 [rows, K], scales: f32 [rows, ceil(K / 128)] -> out: bf16 [rows, K] (contiguous); K % 16 == 0
extern "C" int ifab_dequantize_fp8_block(const void* q, const float* scales, long rows, int K, void* out, void* stream) {
  if (rows < 1 || K < 16 || K % 16) return -1;
  const long items = rows * (K / 16);
  const unsigned blocks = (unsigned)std::min<long>((items + 255) / 256, 148L * 16);
  return launch_chain(dequantize_fp8_block_kernel, dim3(blocks), dim3(256), 0, (cudaStream_t)stream, (const uint8_t*)q, scales, rows, K, (bf16*)out);
}

namespace {
int run_gate_up8(bool streamed, const void* x, long ldx, const void* norm_w, float eps, const int32_t* ids, int T, int D, int F, int topk, int e0, int e_local,
                 const void* w_gu, const float* s_gu, const void* w_shared_gu, const float* s_shared_gu, int Fs, void* act, void* stream) {
  if (D % 16 != 0 || F % 16 != 0 || Fs % 16 != 0 || Fs > F) return -1;
  GateUp8Params p{(const bf16*)x, ldx, (const bf16*)norm_w, eps, ids, T, D, F, topk, e0, e_local,
                  (const uint8_t*)w_gu, s_gu, (const uint8_t*)w_shared_gu, s_shared_gu, Fs, (bf16*)act};
  // by experts, up to eight tokens at a time, where their rows fit beside the rings
  const uintptr_t bits = (uintptr_t)x | (uintptr_t)w_gu | (uintptr_t)w_shared_gu | (uintptr_t)norm_w;
  const size_t room = 232448 - 8192 - XP_RING - XP_RED, row = (size_t)((D * 2 + 127) / 128 * 128 + 16);
  const int at_once = (int)std::min<size_t>(RL_TOKENS, room / row);
  if (streamed && T >= 1 && at_once >= 1 && topk >= 1 && topk <= MAX_TOPK8 && e_local >= 1 && e_local <= RL_EXPERTS && bits % 16 == 0 && ldx % 8 == 0) {
    for (int t0 = 0; t0 < T; t0 += at_once) {
      GateUp8Params q = p;
      q.T = std::min(at_once, T - t0);
      q.x += (long)t0 * ldx;
      q.ids += t0 * topk;
      q.act += (size_t)t0 * (topk + 1) * F;
      const size_t smem = XP_RING + XP_RED + q.T * row;
      // opened for as many tokens as go at once, whatever this step's: by this step's, a thread with fewer tokens would close it for this launch
      if (int rc = opt_in_smem(expert_gate_up_kernel, XP_RING + XP_RED + at_once * row)) return rc;
      if (int rc = (int)cudaFuncSetAttribute(expert_gate_up_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared)) return rc;
      if (int rc = launch_chain(expert_gate_up_kernel, dim3(tc::device_sms()), dim3(256), smem, (cudaStream_t)stream, q)) return rc;
    }
    return 0;
  }
  dim3 grid((F + 15) / 16, T * topk + T);
  const size_t smem = (size_t)D * sizeof(bf16);
  if (int rc = opt_in_smem(moe_gate_up_fp8_kernel, smem)) return rc;
  return launch_chain(moe_gate_up_fp8_kernel, grid, dim3(256), smem, (cudaStream_t)stream, p);
}
}  // namespace

extern "C" int ifab_moe_gate_up_decode_fp8(const void* x, long ldx, const void* norm_w, float eps, const int32_t* ids, int T, int D, int F,
                                           int topk, int e0, int e_local, const void* w_gu, const float* s_gu, const void* w_shared_gu,
                                           const float* s_shared_gu, int Fs, void* act, void* stream) {
  return run_gate_up8(true, x, ldx, norm_w, eps, ids, T, D, F, topk, e0, e_local, w_gu, s_gu, w_shared_gu, s_shared_gu, Fs, act, stream);
}
// The same token by token: for small experts, and for steps whose other kernels stream through L1
extern "C" int ifab_moe_gate_up_tokens_fp8(const void* x, long ldx, const void* norm_w, float eps, const int32_t* ids, int T, int D, int F,
                                           int topk, int e0, int e_local, const void* w_gu, const float* s_gu, const void* w_shared_gu,
                                           const float* s_shared_gu, int Fs, void* act, void* stream) {
  return run_gate_up8(false, x, ldx, norm_w, eps, ids, T, D, F, topk, e0, e_local, w_gu, s_gu, w_shared_gu, s_shared_gu, Fs, act, stream);
}

extern "C" int ifab_moe_down_allreduce_decode_fp8(const void* act, const int32_t* ids, const float* wts, int T, int D, int F, int topk,
                                                  int e0, int e_local, const void* w_down, const float* s_down, const void* w_shared_down,
                                                  const float* s_shared_down, int Fs, const void* residual, long ldr, void* y, long ldy,
                                                  const IfabFabric* fab, void* stream) {
  if (T < 1 || T > 8 || F % 16 != 0 || Fs % 16 != 0 || topk > MAX_TOPK8 || Fs > F) return -1;
  Down8Params p;
  p.act = (const bf16*)act; p.ids = ids; p.wts = wts;
  p.T = T; p.D = D; p.F = F; p.topk = topk; p.e0 = e0; p.e_local = e_local;
  p.w_down = (const uint8_t*)w_down; p.s_down = s_down; p.w_sdown = (const uint8_t*)w_shared_down; p.s_sdown = s_shared_down; p.Fs = Fs;
  p.residual = (const bf16*)residual; p.ldr = ldr; p.y = (bf16*)y; p.ldy = ldy;
  if (int rc = fabric_view(fab, &p.fv)) return rc;
  p.seq = fab->seq; p.done = fab->done;
  if ((size_t)fab->world * T * D * sizeof(uint64_t) > fab->ll_half_bytes) return -3;
  if ((size_t)fab->world * 296 > fab->flag_half_words) return -4;
  cudaStream_t s = (cudaStream_t)stream;
  if (fab->world == 1 && (D + 31) / 32 <= 296 && topk >= 1 && e_local >= 1 && e_local <= RL_EXPERTS && ((uintptr_t)act | (uintptr_t)w_down | (uintptr_t)w_shared_down) % 16 == 0)
    return launch_expert_down(p, s);
  if (T <= 1) return dispatch_down8<1>(p, s);
  if (fab->world == 1) return (D + 31) / 32 <= 296 ? launch_down8<1, 4>(p, s, T) : -2;       // rows as wide as the other forms take
  if (T <= 2) return dispatch_down8<2>(p, s);
  if (T <= 4) return dispatch_down8<4>(p, s);
  return dispatch_down8<8>(p, s);
}
