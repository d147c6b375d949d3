// K1: router. A CTA takes 1, 4 or 8 tokens: it computes the gate logits of every expert, selects
// the top-k experts, turns the selection into combine weights and looks the
// selected experts up in the layer's expert -> cache-slot table.
//
// This replaces the first half of the MoE block forward that the reference
// delegates to its patched transformers fork (gate linear -> softmax -> top-k ->
// optional renormalisation; contract: src/sparse_llm_cache/utils/__init__.py:82-89,
// eval/demo-simulate/transformers-deepseek-moe.py:36-49).
//
// Selection is done on the logits (softmax is monotonic), ties go to the lower
// expert id, and the dot product uses a fixed summation order so that a host
// restatement in float32 reproduces the logits bit for bit:
//   lane j of a warp accumulates the 8-element vectors v with v % 32 == j in
//   ascending v, elements 0..7 in order, acc = acc + w*x (the product of two
//   bf16 values is exact in float32, so fused and unfused multiply-add agree);
//   lanes are then combined by a butterfly over lane ^ 16, 8, 4, 2, 1.
#include <algorithm>

#include "pm_common.cuh"

namespace pm {
namespace {

constexpr int kMaxGateThreads = 512;
constexpr int kMaxExperts = 256;

__device__ __forceinline__ void widen(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

// Logits of EPW expert rows for TOK token rows in shared memory (`stride` vectors apart): a vector of a row is
// widened to float32 once and meets TOK tokens, a vector of a token EPW rows. Each (token, expert) sum runs
// over ascending v inside a lane, the documented order. The next UNROLL vectors of every row are fetched
// before the current ones are used.
template <int TOK, int EPW, int UNROLL>
__device__ __forceinline__ void canonical_dots(const uint4* const (&w)[EPW], const uint4* x, int stride, int nvec, int lane,
                                               float (&acc)[TOK][EPW]) {
#pragma unroll
  for (int t = 0; t < TOK; ++t)
#pragma unroll
    for (int e = 0; e < EPW; ++e) acc[t][e] = 0.f;
  uint4 wv[UNROLL][EPW];
  auto fetch = [&](int v0) {
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      if (v0 + 32 * u < nvec) {
#pragma unroll
        for (int e = 0; e < EPW; ++e) wv[u][e] = __ldg(w[e] + v0 + 32 * u);
      }
  };
  fetch(lane);
  for (int v0 = lane; v0 < nvec; v0 += 32 * UNROLL) {
    float wf[UNROLL][EPW][8];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
#pragma unroll
      for (int e = 0; e < EPW; ++e) widen(wv[u][e], wf[u][e]);
    fetch(v0 + 32 * UNROLL);
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      if (v0 + 32 * u < nvec) {
#pragma unroll
        for (int t = 0; t < TOK; ++t) {
          float xf[8];
          widen(x[(size_t)t * stride + v0 + 32 * u], xf);
#pragma unroll
          for (int e = 0; e < EPW; ++e)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[t][e] = __fmaf_rn(wf[u][e][i], xf[i], acc[t][e]);
        }
      }
  }
#pragma unroll
  for (int t = 0; t < TOK; ++t)
#pragma unroll
    for (int e = 0; e < EPW; ++e)
#pragma unroll
      for (int m = 16; m >= 1; m >>= 1) acc[t][e] += __shfl_xor_sync(0xffffffffu, acc[t][e], m);
}

// One warp turns a token's logits (logit_s[E] = the shared expert's gate) into its k experts and their weights.
// Lane j < k returns the j-th expert.
__device__ __forceinline__ int finish_token(const float* logit_s, int t, int lane, bool has_shared_gate, int E, int k,
                                            int norm_topk, float routed_scale, const int32_t* __restrict__ expert_slot,
                                            int32_t* __restrict__ topk_ids, float* __restrict__ topk_w,
                                            int32_t* __restrict__ topk_slot, float* __restrict__ shared_scale,
                                            float* __restrict__ logits_out) {
  if (logits_out != nullptr)
    for (int e = lane; e < E; e += 32) logits_out[(size_t)t * E + e] = logit_s[e];
  if (has_shared_gate && lane == 0 && shared_scale != nullptr)
    shared_scale[t] = 1.f / (1.f + __expf(-logit_s[E]));

  // Each lane owns experts lane, lane+32, ...
  constexpr int kPerLane = kMaxExperts / 32;
  float v[kPerLane];
  float vmax = -INFINITY;
#pragma unroll
  for (int i = 0; i < kPerLane; ++i) {
    int e = lane + 32 * i;
    v[i] = (e < E) ? logit_s[e] : -INFINITY;
    vmax = fmaxf(vmax, v[i]);
  }
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, m));
  float denom = 0.f;
#pragma unroll
  for (int i = 0; i < kPerLane; ++i)
    if (lane + 32 * i < E) denom += __expf(v[i] - vmax);
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) denom += __shfl_xor_sync(0xffffffffu, denom, m);

  float sel_p = 0.f;   // lane j keeps the probability of the j-th selected expert
  int sel_e = -1;
  float sel_sum = 0.f;
  for (int j = 0; j < k; ++j) {
    float best = -INFINITY;
    int best_e = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
      int e = lane + 32 * i;
      if (e < E && (v[i] > best)) {  // ascending e per lane: strict > keeps the lower id on ties
        best = v[i];
        best_e = e;
      }
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
      float ob = __shfl_xor_sync(0xffffffffu, best, m);
      int oe = __shfl_xor_sync(0xffffffffu, best_e, m);
      if (ob > best || (ob == best && oe < best_e)) {
        best = ob;
        best_e = oe;
      }
    }
    float p = __expf(best - vmax) / denom;
    sel_sum += p;
    if (lane == j) {
      sel_p = p;
      sel_e = best_e;
    }
#pragma unroll
    for (int i = 0; i < kPerLane; ++i)
      if (lane + 32 * i == best_e) v[i] = -INFINITY;
  }
  if (lane < k) {
    float w = sel_p;
    if (norm_topk) w = w / (sel_sum + 1e-20f);
    w *= routed_scale;
    topk_ids[(size_t)t * k + lane] = sel_e;
    topk_w[(size_t)t * k + lane] = w;
    if (topk_slot != nullptr)
      topk_slot[(size_t)t * k + lane] = (expert_slot != nullptr && sel_e < E) ? expert_slot[sel_e] : -1;
  }
  return sel_e;
}

// TOK tokens per CTA, EPW expert rows per warp at a time (see launch_gate_topk for the choice).
template <int TOK, int EPW, int UNROLL>
__global__ void __launch_bounds__(kMaxGateThreads)
gate_topk_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w_gate,
                 const float* __restrict__ bias, const __nv_bfloat16* __restrict__ w_shared_gate,
                 int T, int H, int E, int k, int norm_topk, float routed_scale,
                 const int32_t* __restrict__ expert_slot, int32_t* __restrict__ topk_ids,
                 float* __restrict__ topk_w, int32_t* __restrict__ topk_slot,
                 float* __restrict__ shared_scale, float* __restrict__ logits_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];  // TOK rows of H bf16
  __shared__ float logit_all[TOK * (kMaxExperts + 1)];
  wait_for_predecessor();

  const int t0 = blockIdx.x * TOK;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwarp = blockDim.x / 32;
  const int nvec = H / 8;
  const int n_tok = min(TOK, T - t0);

  uint4* xs = reinterpret_cast<uint4*>(smem_raw);
  {
    const uint4* xp = reinterpret_cast<const uint4*>(x + (size_t)t0 * H);
    for (int idx = threadIdx.x; idx < TOK * nvec; idx += blockDim.x)
      xs[idx] = idx < n_tok * nvec ? __ldg(xp + idx) : make_uint4(0, 0, 0, 0);
  }
  __syncthreads();
  const int n_rows = E + (w_shared_gate != nullptr ? 1 : 0);
  for (int e0 = warp * EPW; e0 < n_rows; e0 += nwarp * EPW) {
    const uint4* wp[EPW];
#pragma unroll
    for (int i = 0; i < EPW; ++i) {
      const int e = min(e0 + i, n_rows - 1);
      wp[i] = (e < E) ? reinterpret_cast<const uint4*>(w_gate + (size_t)e * H) : reinterpret_cast<const uint4*>(w_shared_gate);
    }
    float d[TOK][EPW];
    canonical_dots<TOK, EPW, UNROLL>(wp, xs, nvec, nvec, lane, d);
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < EPW; ++i) {
        const int e = e0 + i;
        if (e >= n_rows) break;
        const bool has_bias = e < E && bias != nullptr;
        const float bv = has_bias ? bias[e] : 0.f;
#pragma unroll
        for (int tt = 0; tt < TOK; ++tt) logit_all[tt * (E + 1) + e] = has_bias ? d[tt][i] + bv : d[tt][i];
      }
    }
  }
  __syncthreads();

  for (int tt = warp; tt < n_tok; tt += nwarp)  // warp tt finishes token t0 + tt
    finish_token(logit_all + tt * (E + 1), t0 + tt, lane, w_shared_gate != nullptr, E, k, norm_topk, routed_scale, expert_slot,
                 topk_ids, topk_w, topk_slot, shared_scale, logits_out);
}

// Router and permutation of a decode batch in ONE launch: a cluster of eight CTAs splits the expert rows (one SM
// alone takes 4 us just to read a 64 x 2048 router matrix out of L2), every CTA sends its logits to the first one
// through distributed shared memory, and that one selects the experts and lays the T * k pairs out per expert.
// Same sums, in the same order, as gate_topk_kernel; same layout as the permutation kernels. A pass of one token over 64
// experts went from 55.1 to 45.9 us with it; in two launches (CUDA graph) the router took 9.2 us and the permutation 3.2.
constexpr int kRouteCtas = 8, kRouteThreads = 512, kRouteMaxTokens = 16, kRouteMaxTopK = 16;

template <int TOK>
__global__ void __cluster_dims__(kRouteCtas, 1, 1) __launch_bounds__(kRouteThreads)
route_small_kernel(const __grid_constant__ RouteArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];  // the token rows, padded to a multiple of TOK
  __shared__ float logit_all[kRouteMaxTokens * (kMaxExperts + 1)];
  __shared__ int ids_s[kRouteMaxTokens * kRouteMaxTopK];
  __shared__ int cnt[kMaxExperts];
  __shared__ int off[kMaxExperts + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int T = a.T, E = a.E, k = a.k, nvec = a.H / 8, R = T * k;
  const int n_rows = E + (a.w_shared_gate != nullptr ? 1 : 0);
  const int groups = (T + TOK - 1) / TOK;
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // waited for before the first remote store
  wait_for_predecessor();

  uint4* xs = reinterpret_cast<uint4*>(smem_raw);
  for (int idx = tid; idx < groups * TOK * nvec; idx += kRouteThreads)
    xs[idx] = idx < T * nvec ? __ldg(reinterpret_cast<const uint4*>(a.x) + idx) : make_uint4(0, 0, 0, 0);
  if (rank == 0)
    for (int e = tid; e < E; e += kRouteThreads) cnt[e] = 0;
  if (rank == 1)  // work without a dependency, beside the dot products
    for (int i = tid; i < a.zero_n; i += kRouteThreads) a.zero_words[i] = 0;
  if (rank == 2)
    for (int i = tid; i < a.tail_rows; i += kRouteThreads) a.row_token[R + i] = i % T;
  __syncthreads();

  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // the first CTA runs: its shared memory may be written

  uint32_t logit0;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(logit0) : "r"((uint32_t)__cvta_generic_to_shared(logit_all)));
  const int per = (n_rows + kRouteCtas - 1) / kRouteCtas, first = rank * per;
  const int mine = min(per, n_rows - first);
  for (int task = warp; task < mine * groups; task += kRouteThreads / 32) {
    const int g = task % groups, e = first + task / groups;
    const uint4* wp[1] = {e < E ? reinterpret_cast<const uint4*>(a.w_gate + (size_t)e * a.H)
                                : reinterpret_cast<const uint4*>(a.w_shared_gate)};
    float d[TOK][1];
    canonical_dots<TOK, 1, 4>(wp, xs + (size_t)g * TOK * nvec, nvec, nvec, lane, d);
    float v = d[0][0];
#pragma unroll
    for (int t = 1; t < TOK; ++t)
      if (lane == t) v = d[t][0];
    if (e < E && a.bias != nullptr) v = v + a.bias[e];
    if (lane < TOK && g * TOK + lane < T)
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(logit0 + 4u * (uint32_t)((g * TOK + lane) * (E + 1) + e)), "f"(v)
                   : "memory");
    __syncwarp();
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (rank != 0) return;

  for (int t = warp; t < T; t += kRouteThreads / 32) {
    const int e = finish_token(logit_all + t * (E + 1), t, lane, a.w_shared_gate != nullptr, E, k, a.norm_topk,
                               a.routed_scale, a.expert_slot, a.topk_ids, a.topk_w, a.topk_slot, a.shared_scale, nullptr);
    if (lane < k) ids_s[t * k + lane] = e;
  }
  __syncthreads();
  // pair i's place inside its expert = the pairs of the expert before it (R is at most 256)
  int e = -1, before = 0;
  if (tid < R) {
    e = ids_s[tid];
    if (e < 0 || e >= E) {  // only where no logit compares (NaN): dropped and flagged, as by the permutation
      e = -1;
      a.pos[tid] = -1;
      if (a.err_flag != nullptr) atomicExch(a.err_flag, 1);
    } else {
      for (int j = 0; j < tid; ++j) before += ids_s[j] == e;
      atomicAdd(&cnt[e], 1);
    }
  }
  __syncthreads();
  if (warp == 0) {
    int run = 0;
    for (int c = 0; c < E; c += 32) {
      const int n = c + lane < E ? cnt[c + lane] : 0;
      int incl = n;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
      }
      if (c + lane < E) off[c + lane] = run + incl - n;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) off[E] = run;
  }
  __syncthreads();
  for (int i = tid; i < E; i += kRouteThreads) a.counts[i] = cnt[i];
  for (int i = tid; i <= E; i += kRouteThreads) a.offsets[i] = off[i];
  for (int i = off[E] + tid; i < R; i += kRouteThreads) a.row_token[i] = 0;  // rows that no pair takes
  if (e >= 0) {
    const int p = off[e] + before;
    a.row_token[p] = tid / k;
    a.pos[tid] = p;
  }
}

template <int TOK, int EPW, int UNROLL>
cudaError_t launch_gate(const __nv_bfloat16* x, const __nv_bfloat16* w_gate, const float* bias,
                        const __nv_bfloat16* w_shared_gate, int T, int H, int E, int k, int norm_topk,
                        float routed_scale, const int32_t* expert_slot, int32_t* topk_ids, float* topk_w,
                        int32_t* topk_slot, float* shared_scale, float* logits_out, cudaStream_t s) {
  const int n_rows = E + (w_shared_gate != nullptr ? 1 : 0);
  const int warps = std::min(kMaxGateThreads / 32, (n_rows + EPW - 1) / EPW);
  const size_t smem = (size_t)TOK * H * 2;
  auto kern = gate_topk_kernel<TOK, EPW, UNROLL>;
  static SmemOptIn once;
  if (smem > 32 * 1024) {
    cudaError_t e = opt_in_smem(once, kern);
    if (e != cudaSuccess) return e;
  }
  return launch_behind(kern, (T + TOK - 1) / TOK, warps * 32, smem, s, x, w_gate, bias, w_shared_gate, T, H, E, k, norm_topk,
                       routed_scale, expert_slot, topk_ids, topk_w, topk_slot, shared_scale, logits_out);
}

size_t route_small_smem(int T, int H) { return (size_t)(T > 1 ? (T + 3) / 4 * 4 : 1) * H * 2; }

}  // namespace

bool route_small_usable(int T, int H) { return T <= kRouteMaxTokens && route_small_smem(T, H) <= 160 * 1024; }

cudaError_t launch_route_small(const RouteArgs& a, cudaStream_t s) {
  const size_t smem = route_small_smem(a.T, a.H);
  auto kern = a.T > 1 ? route_small_kernel<4> : route_small_kernel<1>;
  static SmemOptIn once[2];
  if (smem > 16 * 1024) {  // beside 19 KB of static shared memory
    cudaError_t e = opt_in_smem(once[a.T > 1], kern);
    if (e != cudaSuccess) return e;
  }
  return launch_behind(kern, kRouteCtas, kRouteThreads, smem, s, a);
}

cudaError_t launch_gate_topk(const __nv_bfloat16* x, const __nv_bfloat16* w_gate, const float* bias,
                             const __nv_bfloat16* w_shared_gate, int T, int H, int E, int k, int norm_topk,
                             float routed_scale, const int32_t* expert_slot, int32_t* topk_ids, float* topk_w,
                             int32_t* topk_slot, float* shared_scale, float* logits_out, cudaStream_t s) {
  if (T <= 0) return cudaSuccess;
  auto go = [&](auto launch) {
    return launch(x, w_gate, bias, w_shared_gate, T, H, E, k, norm_topk, routed_scale, expert_slot, topk_ids, topk_w,
                  topk_slot, shared_scale, logits_out, s);
  };
  // Up to two waves of one CTA per SM a token has a CTA to itself (most loads in flight); then 4, and from
  // about three waves of 4 on, 8 tokens share a CTA's reads of the router matrix. Few experts: one or two
  // rows per warp, so that a CTA still has enough warps.
  const bool few = E <= 16;
  if (T <= 296 || (size_t)8 * H * 2 > 160 * 1024) return few ? go(launch_gate<1, 1, 4>) : go(launch_gate<1, 4, 1>);
  if (T < 1776) return few ? go(launch_gate<4, 1, 4>) : go(launch_gate<4, 4, 1>);
  return few ? go(launch_gate<8, 1, 2>) : go(launch_gate<8, 4, 1>);
}

}  // namespace pm
