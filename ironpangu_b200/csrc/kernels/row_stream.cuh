// Products of one to eight rows with a weight matrix, the core of the decode linears:  out[t][n] = sum_k x[t][k] W[n][k].
//
// Bound by the stream of W (2 bytes a weight, used once), so what matters is that HBM never waits. One CTA an SM takes an equal share of the rows of W
// (N / 148 of them, whatever N is) and its eight warps an eighth of K each; every warp streams its share through a ring of its own in shared memory
// (cp.async in whole 128-byte lines, no barrier among the warps). The ring is filled before the wait for the preceding kernel, and the next linear's CTA is on the SM
// while this one multiplies, sums up and drains, so that its first 10 to 14 MB are on the way. With the loads in registers and grids of two CTAs an SM the next
// kernel found no room before the last wave ended. Bulk copies in place of cp.async reached 4.0 TB/s (a CTA of eight rows of 2 KB a copy) against 6.0.
// Products are m16n8k16 with the rows of x as rows of A and eight rows of W as columns of B: a lane's 16 bytes of W are the B operands of two of them. K is
// permuted alike in A and B (a lane's eight consecutive columns are 2q, 2q+1, 2q+8, 2q+9 of both products), so nothing is shuffled. (Rows of W as the sixteen rows of A
// halve the products, but tiles of sixteen rows waste more of the ring: 2B layer 23.4 -> 23.7 us, 8B 81 -> 91.) Each product of 16 terms
// is added to its f32 sum outside the tensor core (which cuts off what it adds up), and the eight warps' sums are added in one order: against 64 bits 7.4e-8 off at
// K 2048 and 8.6e-8 at 6144, where FMAs along a lane were 8.0e-8 and 1.1e-7. What a row of x gets depends on nothing but that row: its bits are the same whatever rows are
// beside it.
// The four linears of a layer (with their norms, residuals and gated unit) one after the other, us before -> after, by rows of x 1 / 2 / 8: width 1024 and
// feed-forward 4096 (31 MB) 14.8 / 22.5 / 71 -> 13.1 / 15.4 / 15.3; 2048 and 6144 (97 MB) 26.7 / 36 / 108 -> 23.4 / 25.6 / 28.2; 4096 and 16384 (487 MB) 91.5 / 118 / -
// -> 81 / 82 / 92.
#pragma once
#include "mma16816.cuh"
#include "tc_common.cuh"

namespace ifab {

constexpr int RS_WARPS = 8, RS_STEPS = 4;                      // warps of a CTA; steps of 32 columns in a stage of a warp's ring
constexpr int RS_STAGE = RS_STEPS * 512;                       // bytes: eight rows of W by 128 columns

// 16 bytes that the preceding kernel has written (volatile: issued where it stands, ahead of what uses the ones before it)
__device__ __forceinline__ uint4 ld_row16(const bf16* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_shared16(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared16(uint32_t at, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// A CTA's share of the product: results lo <= n < hi of N. PLAIN: of row n of W [N, K]; GATED: of rows n and N + n of W [2 N, K]; PAIRS: of the two rows that a
// rotation turns into one another, n + n / half * half and the one half behind, of W [2 N, K]
enum class Rows { PLAIN, GATED, PAIRS };
struct RowShare {
  const bf16* w;
  int N, K, lo, hi, half;
};

// MR: most rows of x. TB: tiles of eight rows of W that are summed up at a time (GATED and PAIRS: half of them first rows, the other half the second ones).
// DEPTH: stages of a ring. XS: bytes for rows of x
template <int MR, int TB, int DEPTH, int XS, Rows KIND>
struct RowStream {
  static constexpr bool TWO = KIND != Rows::PLAIN;
  static constexpr int PER = TWO ? 2 : 1, ROWS = 8 * TB / PER;      // outputs of a block of tiles
  static constexpr int RING = RS_WARPS * DEPTH * RS_STAGE, RED = RS_WARPS * TB * MR * 8 * 4, SMEM = RING + RED + XS;

  RowShare s;
  uint32_t ring, xs;             // this warp's; rows of x, `pitch` bytes apart
  float* red;                    // [warps][TB][MR][8 rows of W]
  int warp, lane, pitch;
  int steps, chunk, chunks;      // steps of 32 columns of a warp in a stage, columns of all warps' stages, stages along K
  int col;                       // first column of this warp in a chunk
  // the next stage to be requested: block, chunk, tile, tiles of the block; this lane's piece of it: row lane / 8 of the tile and the fourth one behind, 16-byte
  // piece lane % 8 of 128 bytes
  int pb, pk, pt, pn;
  const bf16* src;               // this lane's piece of the block's first tile

  __device__ __forceinline__ int tiles_of(int lo) const { return PER * ((min(ROWS, s.hi - lo) + 7) / 8); }
  __device__ __forceinline__ const bf16* piece(int lo, int k) const {
    return s.w + (long)min(lo + (lane >> 3), s.N - 1) * s.K + k * chunk + col + (lane & 7) * 8;
  }
  __device__ __forceinline__ void request(int at) {
    if (pb < s.hi) {
      const int r = pb + pt / PER * 8 + (lane >> 3), left = min(steps * 32, s.K - pk * chunk - col) - (lane & 7) * 8;
      const bf16 *from = src + (long)(pt / PER * 8 + (KIND == Rows::GATED && (pt & 1) ? s.N : 0)) * s.K, *from4 = from + 4l * s.K;
      if (KIND == Rows::PAIRS) {
        const int a = min(r, s.N - 1), b = min(r + 4, s.N - 1), second = pt & 1 ? s.half : 0;
        const bf16* at_col = s.w + pk * chunk + col + (lane & 7) * 8;
        from = at_col + (long)(a + a / s.half * s.half + second) * s.K;
        from4 = at_col + (long)(b + b / s.half * s.half + second) * s.K;
      }
      // a piece lies where its reader's accesses meet no bank twice
      const uint32_t dst = ring + at * RS_STAGE + (lane >> 3) * 128 + (((lane & 7) ^ (lane >> 3)) << 4), dst4 = dst ^ 64;
      const bool row = r < s.hi, row4 = r + 4 < s.hi;
#pragma unroll
      for (int h = 0; h < RS_STEPS / 2; ++h) {
        const bool in = row && h * 64 < left, in4 = row4 && h * 64 < left;
        copy16(dst + h * 1024, in ? from + h * 64 : s.w, in);
        copy16(dst4 + h * 1024 + 512, in4 ? from4 + h * 64 : s.w, in4);
      }
      if (++pt == pn) {
        pt = 0;
        if (++pk == chunks) {
          pk = 0;
          pb += ROWS;
          pn = tiles_of(pb);
        }
        src = piece(pb, pk);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // all threads, before the wait for the preceding kernel: W is written by no kernel of the stream
  __device__ __forceinline__ void start(const RowShare& share, unsigned char* smem) {
    s = share;
    warp = threadIdx.x >> 5;
    lane = threadIdx.x & 31;
    ring = smem_addr(smem) + warp * DEPTH * RS_STAGE;
    red = reinterpret_cast<float*>(smem + RING);
    xs = smem_addr(smem) + RING + RED;
    pitch = (s.K * 2 + 127) / 128 * 128 + 16;
    chunks = (s.K + RS_WARPS * RS_STEPS * 32 - 1) / (RS_WARPS * RS_STEPS * 32);
    steps = ((s.K + chunks * RS_WARPS * 64 - 1) / (chunks * RS_WARPS * 64)) * 2;
    chunk = steps * RS_WARPS * 32;
    col = warp * steps * 32;
    pb = s.lo;
    pk = pt = 0;
    pn = tiles_of(pb);
    src = piece(pb, 0);
#pragma unroll 1
    for (int i = 0; i < DEPTH; ++i) request(i);
  }
  // columns of step u of this lane's operands, within the warp's of a chunk
  __device__ __forceinline__ int at_step(int u) const { return (u >> 1) * 64 + (lane & 3) * 16 + (u & 1) * 8; }
  __device__ __forceinline__ bool fits(int T) const { return T * pitch <= XS; }
  __device__ __forceinline__ bool first_result(int T, int* t, int* n) const {
    const int c = threadIdx.x & 7, j = threadIdx.x >> 3, p = j / T;
    *t = j - p * T;
    *n = s.lo + p * 8 + c;
    return p < tiles_of(s.lo) / PER && *n < s.hi;
  }

  // `x.load(k, raw)` requests this lane's operands of chunk k (row lane / 4 of x, columns k chunk + col + at_step(u) on), `x.operand(k, raw, a)` has them as bf16;
  // `out(t, n, v, u, first)` takes a result (u: of row N + n; first: it is the thread's first, which first_result() names ahead). T: rows of x.
  template <class X, class Out>
  __device__ __forceinline__ void run(X& x, int T, Out& out) {
    typename X::Raw raw;
    x.load(*this, 0, raw);
    int slot = 0;
    const uint32_t even = ring + (lane >> 2) * 128 + (((lane & 3) * 2 ^ (lane >> 2)) << 4);
#pragma unroll 1
    for (int lo = s.lo; lo < s.hi; lo += ROWS) {
      const int tiles = tiles_of(lo);
      float2* sums = reinterpret_cast<float2*>(red + warp * TB * MR * 8 + (lane >> 2) * 8 + (lane & 3) * 2);      // this lane's, MR * 8 floats a tile
      const bool mine = MR == 8 || (lane >> 2) < MR;
#pragma unroll 1
      for (int k = 0; k < chunks; ++k) {
        uint4 a[RS_STEPS];
        x.operand(*this, k, raw, a);
        x.load(*this, k + 1 < chunks ? k + 1 : 0, raw);
#pragma unroll 1
        for (int t = 0; t < tiles; ++t) {
          asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
          __syncwarp();
          const uint32_t at = even + slot * RS_STAGE;
          uint4 b[RS_STEPS];
#pragma unroll
          for (int u = 0; u < RS_STEPS; ++u) b[u] = ld_shared16((u & 1 ? at ^ 16 : at) + (u >> 1) * 1024);
          float2 acc = k && mine ? sums[t * MR * 4] : make_float2(0.f, 0.f), part[RS_STEPS];
#pragma unroll
          for (int u = 0; u < RS_STEPS; ++u) {
            float d[4], e[4];
            mma16816_alone(d, a[u].x, 0u, a[u].y, 0u, b[u].x, b[u].y);
            mma16816_alone(e, a[u].z, 0u, a[u].w, 0u, b[u].z, b[u].w);
            part[u] = make_float2(d[0] + e[0], d[1] + e[1]);
          }
          __syncwarp();            // the stage is read
          request(slot);
          acc.x += (part[0].x + part[1].x) + (part[2].x + part[3].x);
          acc.y += (part[0].y + part[1].y) + (part[2].y + part[3].y);
          if (mine) sums[t * MR * 4] = acc;
          slot = slot + 1 == DEPTH ? 0 : slot + 1;
        }
      }
      __syncthreads();
      const int n_out = tiles / PER * 8 * T;
      for (int i = threadIdx.x; i < n_out; i += RS_WARPS * 32) {
        const int c = i & 7, j = i >> 3, p = j / T, t = j - p * T, n = lo + p * 8 + c;
        if (n >= s.hi) continue;
        const float* from = red + (p * PER * MR + t) * 8 + c;
        auto sum = [&](const float* f) {
          constexpr int W = TB * MR * 8;
          return ((f[0] + f[W]) + (f[2 * W] + f[3 * W])) + ((f[4 * W] + f[5 * W]) + (f[6 * W] + f[7 * W]));
        };
        out(t, n, sum(from), TWO ? sum(from + MR * 8) : 0.f, lo == s.lo && i == (int)threadIdx.x);
      }
      if (lo + ROWS < s.hi) __syncthreads();
    }
  }
};

// rows of x in bf16, as they are or RMS-normalised: bf16(x rsqrt(mean(x^2) + eps) (w or 1 + w)). Where they fit they lie in shared memory, having been loaded in
// whole rows once (every SM reads all of x at the same time: in the pieces that the products take, 64 bytes of each row, eight rows of 2048 columns took
// 2.5 us); otherwise a lane reads its pieces from L2, one chunk ahead.
template <int MR, bool NORM>
struct BfRows {
  struct Raw {
    uint4 x[RS_STEPS], gain[NORM ? RS_STEPS : 1];
  };
  static constexpr int NV = MR == 8 ? 8 : 2;         // pieces of a row that a thread holds at a time
  static constexpr int NT = MR == 8 ? 32 : RS_WARPS * 32;      // threads that share a row: a warp, or all
  const bf16* x; long ldx;
  const bf16* norm_w; float eps; int zero_centered, T;
  float inv;
  bool staged;
  uint4 gain[NORM ? NV : 1];

  __device__ __forceinline__ uint4 scaled(const uint4& v, const uint4& w, float by) const {
    float f[8], g[8];
    unpack8(v, f);
    unpack8(w, g);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = f[i] * by * (zero_centered ? 1.f + g[i] : g[i]);
    return pack8(f);
  }
  __device__ __forceinline__ int first() const { return MR == 8 ? threadIdx.x & 31 : threadIdx.x; }
  // before the wait: gains are weights
  template <class S>
  __device__ __forceinline__ void early(const S& s) {
    staged = s.fits(T);
    if constexpr (NORM) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = first() + i * NT;
        gain[i] = c * 8 < s.s.K ? *reinterpret_cast<const uint4*>(norm_w + c * 8) : make_uint4(0, 0, 0, 0);
      }
    }
  }
  // the warps that multiply, after the wait; `sums`: [warps][8] floats of shared memory. MR 8: a warp a row; otherwise all of them every row
  template <class S>
  __device__ __forceinline__ void prepare(const S& s, float* sums) {
    const int pieces = s.s.K >> 3;
    if (!NORM && !staged) return;
#pragma unroll
    for (int r = 0; r < (MR == 8 ? 1 : MR); ++r) {
      const int t = MR == 8 ? s.warp : r;
      if (t >= T) break;
      const bf16* row = x + (long)t * ldx;
      const uint32_t to = s.xs + t * s.pitch;
      // The sum of squares in one order whatever the threads: of 256 threads' pieces, 32 threads at a time. A warp alone has the pieces of eight warps.
      constexpr int NS = MR == 8 ? NV : 1;
      float ss[NS] = {};
#pragma unroll 1
      for (int c0 = first(); c0 < pieces; c0 += NV * NT) {
        uint4 v[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          v[i] = make_uint4(0, 0, 0, 0);
          if (c0 + i * NT < pieces) v[i] = ld_row16(row + (c0 + i * NT) * 8);
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          if (staged && c0 + i * NT < pieces) st_shared16(to + (c0 + i * NT) * 16, v[i]);
          if (NORM) {
            float f[8];
            unpack8(v[i], f);
#pragma unroll
            for (int e = 0; e < 8; ++e) ss[i % NS] += f[e] * f[e];
          }
        }
      }
      if (NORM) {
#pragma unroll
        for (int i = 0; i < NS; ++i) ss[i] = warp_sum(ss[i]);
        if (MR == 8) {
#pragma unroll
          for (int i = 1; i < NS; ++i) ss[0] += ss[i];
        }
        if (s.lane == 0) sums[MR == 8 ? t : s.warp * 8 + t] = ss[0];
      }
    }
    if (NORM) {
      if (MR == 8 && staged) __syncwarp();
      else __syncthreads();
      if (!staged) {
        inv = scale_of(s, sums, min(s.lane >> 2, T - 1));
        return;
      }
#pragma unroll
      for (int r = 0; r < (MR == 8 ? 1 : MR); ++r) {
        const int t = MR == 8 ? s.warp : r;
        if (t >= T) break;
        const float by = scale_of(s, sums, t);
        const uint32_t to = s.xs + t * s.pitch;
#pragma unroll 1
        for (int c0 = first(); c0 < pieces; c0 += NV * NT)
#pragma unroll
          for (int i = 0; i < NV; ++i) {
            const int c = c0 + i * NT;
            if (c < pieces) st_shared16(to + c * 16, scaled(ld_shared16(to + c * 16), c0 == first() ? gain[i] : *reinterpret_cast<const uint4*>(norm_w + c * 8), by));
          }
      }
    }
    __syncthreads();
  }
  template <class S>
  __device__ __forceinline__ float scale_of(const S& s, const float* sums, int t) const {
    float sum = sums[t];
    if (MR != 8) {
#pragma unroll
      for (int w = 1; w < RS_WARPS; ++w) sum += sums[w * 8 + t];
    }
    return rsqrtf(sum / (float)s.s.K + eps);
  }
  template <class S>
  __device__ __forceinline__ bool has(const S& s, int k, int u) const {
    return (s.lane >> 2) < T && u < s.steps && k * s.chunk + s.col + s.at_step(u) < s.s.K;
  }
  template <class S>
  __device__ __forceinline__ void load(const S& s, int k, Raw& raw) const {
    if (staged) return;
    const int c0 = k * s.chunk + s.col;
#pragma unroll
    for (int u = 0; u < RS_STEPS; ++u) {
      raw.x[u] = make_uint4(0, 0, 0, 0);
      if (has(s, k, u)) raw.x[u] = ld_row16(x + (long)(s.lane >> 2) * ldx + c0 + s.at_step(u));
      if (NORM) {
        raw.gain[u] = make_uint4(0, 0, 0, 0);
        if (has(s, k, u)) raw.gain[u] = ld_row16(norm_w + c0 + s.at_step(u));
      }
    }
  }
  template <class S>
  __device__ __forceinline__ void operand(const S& s, int k, const Raw& raw, uint4 (&a)[RS_STEPS]) const {
    if (staged) {
      const uint32_t at = s.xs + (s.lane >> 2) * s.pitch + (k * s.chunk + s.col) * 2;
#pragma unroll
      for (int u = 0; u < RS_STEPS; ++u) {
        a[u] = make_uint4(0, 0, 0, 0);
        if (has(s, k, u)) a[u] = ld_shared16(at + s.at_step(u) * 2);
      }
      return;
    }
#pragma unroll
    for (int u = 0; u < RS_STEPS; ++u) a[u] = NORM ? scaled(raw.x[u], raw.gain[u], inv) : raw.x[u];
  }
};

}  // namespace ifab
