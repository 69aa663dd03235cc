// The routes of a step's tokens as a list of experts, each with the tokens that chose it: what the expert kernels go through when every expert's weights are read once for all
// of its tokens.
//
// Experts come in ascending order, so that what a token gets is added up in an order of its own choices, whatever tokens are beside it. A token that names an expert
// twice has an entry of its own for the second time, at the end.
#pragma once
#include "common.cuh"

namespace ifab {

constexpr int RL_TOKENS = 8, RL_ROUTES = RL_TOKENS * 16, RL_EXPERTS = 1024;

struct RouteList {
  int n;                                    // entries
  uint16_t expert[RL_ROUTES];               // of the local ones, from 0
  int8_t slot[RL_ROUTES][RL_TOKENS];        // which of a token's choices it is; -1: not among them
  // scratch
  int ids[RL_ROUTES];
  uint32_t bits[RL_EXPERTS / 32];
  int ahead[RL_EXPERTS / 32], again;
};

// all threads of a CTA of 256 (ids are there: behind the wait for the router); ends with a barrier
__device__ __forceinline__ void list_routes(RouteList& r, const int32_t* ids, int T, int topk, int e0, int e_local) {
  const int tid = threadIdx.x, routes = T * topk;
  for (int i = tid; i < RL_ROUTES * RL_TOKENS / 4; i += 256) reinterpret_cast<uint32_t*>(r.slot)[i] = 0xffffffffu;
  if (tid < RL_EXPERTS / 32) r.bits[tid] = 0;
  if (tid == 0) r.again = 0;
  const int e = tid < routes ? ids[tid] - e0 : -1;
  if (tid < routes) r.ids[tid] = e;
  __syncthreads();
  const int t = tid / topk, s = tid - t * topk;
  bool live = tid < routes && e >= 0 && e < e_local, twice = false;
  if (live) {
    for (int i = t * topk; i < tid; ++i) twice |= r.ids[i] == e;
    if (twice) atomicAdd(&r.again, 1);
    else atomicOr(&r.bits[e >> 5], 1u << (e & 31));
  }
  __syncthreads();
  if (tid < 32) {
    const int mine = __popc(r.bits[tid]);
    int sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (tid >= o) sum += v;
    }
    r.ahead[tid] = sum - mine;
    if (tid == 31) r.n = sum;
  }
  __syncthreads();
  if (live && !twice) {
    const int at = r.ahead[e >> 5] + __popc(r.bits[e >> 5] & ((1u << (e & 31)) - 1u));
    r.expert[at] = (uint16_t)e;
    r.slot[at][t] = (int8_t)s;
  }
  if (r.again && tid == 0) {
    int n = r.n;
    for (int i = 0; i < routes; ++i) {
      const int ei = r.ids[i], first = i / topk * topk;
      if (ei < 0 || ei >= e_local) continue;
      bool seen = false;
      for (int j = first; j < i; ++j) seen |= r.ids[j] == ei;
      if (!seen) continue;
      r.expert[n] = (uint16_t)ei;
      r.slot[n][i / topk] = (int8_t)(i - first);
      ++n;
    }
    r.again = n;                            // read below, when everybody has passed the test above
  }
  __syncthreads();
  if (tid == 0 && r.again) r.n = r.again;
  __syncthreads();
}

}  // namespace ifab
