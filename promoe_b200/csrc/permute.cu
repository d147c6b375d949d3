// K2: token permutation. Turns the [T, k] routing table into per-expert
// contiguous row ranges: counts[E], offsets[E+1], row_token[R] (the token each
// permuted row reads) and pos[R] (where routed pair (t, j) landed). The order
// inside one expert is ascending in t*k + j, so the result is deterministic.
//
// The reference has no such step: its patched MoE block loops over experts in
// Python and indexes the hidden states per expert (contract:
// eval/demo-simulate/transformers-deepseek-moe.py:41-48). counts[] is also what
// the host reads back to form the unique expert list it reports to the cache
// (src/cpp_worker/prefetcher.cpp:188-202).
#include "pm_common.cuh"

namespace pm {
namespace {

constexpr int kPermThreads = 1024;  // pairs placed at a time: one per thread
constexpr int kPermWarps = kPermThreads / 32;
constexpr int kMaxExperts = 256;

// off[e] = sum of tot[0 .. e), off[E] = sum of all. One warp.
__device__ __forceinline__ void scan_experts(const int* tot, int* off, int E) {
  const int lane = threadIdx.x & 31;
  int run = 0;
  for (int c = 0; c < E; c += 32) {
    const int n = c + lane < E ? tot[c + lane] : 0;
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

// Places up to 1024 pairs (thread's pair i of expert e, -1 = none) behind base[e] in shared memory and advances
// base. Inside an expert the order is ascending in the pair's index: the lanes of a warp that hold the same
// expert find each other with one match instruction, and a pair's place is base + the expert's pairs in
// lower warps + the lower lanes. (One warp per expert scanning all pairs took 34 us for 3108 pairs over 60
// experts, now 8 us; 555 us for 49152 over 64, now 90 us.)
__device__ __forceinline__ void place_pairs(int i, int e, int k, int E, int* base, unsigned short (*wcnt)[kMaxExperts],
                                            int32_t* __restrict__ row_token, int32_t* __restrict__ pos) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int x = tid; x < kPermWarps * kMaxExperts / 2; x += kPermThreads) reinterpret_cast<uint32_t*>(wcnt)[x] = 0;
  __syncthreads();
  const unsigned peers = __match_any_sync(0xffffffffu, e);
  const int before = __popc(peers & ((1u << lane) - 1u));
  if (e >= 0 && before == 0) wcnt[warp][e] = (unsigned short)__popc(peers);
  __syncthreads();
  int placed = 0;  // thread e: pairs of expert e
  if (tid < E) {
#pragma unroll
    for (int w = 0; w < kPermWarps; ++w) {
      const int n = wcnt[w][tid];
      wcnt[w][tid] = (unsigned short)placed;
      placed += n;
    }
  }
  __syncthreads();
  if (e >= 0) {
    const int p = base[e] + wcnt[warp][e] + before;
    row_token[p] = i / k;
    pos[i] = p;
  }
  __syncthreads();
  if (tid < E) base[tid] += placed;
}

// Expert of pair i, -1 for a pair that is dropped: padding (-1, silently) or an id outside [0, E), which is flagged.
__device__ __forceinline__ int expert_of(const int32_t* __restrict__ topk_ids, int i, int R, int E, int32_t* err_flag) {
  if (i >= R) return -1;
  const int e = topk_ids[i];
  if (e >= 0 && e < E) return e;
  if (e != -1 && err_flag != nullptr) atomicExch(err_flag, 1);
  return -1;
}

// One CTA, any number of pairs: counts, offsets, then 1024 pairs at a time.
__global__ void __launch_bounds__(kPermThreads)
permute_kernel(const int32_t* __restrict__ topk_ids, int R, int k, int E, int32_t* __restrict__ counts,
               int32_t* __restrict__ offsets, int32_t* __restrict__ row_token,
               int32_t* __restrict__ pos, int32_t* __restrict__ err_flag, int tail_rows, int T,
               int32_t* __restrict__ zero_words, int zero_n) {
  __shared__ unsigned short wcnt[kPermWarps][kMaxExperts];
  __shared__ int cnt[kMaxExperts];
  __shared__ int base[kMaxExperts + 1];
  const int tid = threadIdx.x;
  wait_for_predecessor();
  for (int e = tid; e < E; e += kPermThreads) cnt[e] = 0;
  for (int i = tid; i < zero_n; i += kPermThreads) zero_words[i] = 0;
  // Rows after the R routed ones belong to the shared experts: every token once per shared expert.
  for (int i = tid; i < tail_rows; i += kPermThreads) row_token[R + i] = i % T;
  __syncthreads();
  for (int i = tid; i < R; i += kPermThreads) {
    const int e = expert_of(topk_ids, i, R, E, err_flag);
    if (e >= 0) atomicAdd(&cnt[e], 1);
    else pos[i] = -1;  // the position must not keep an old value
  }
  __syncthreads();
  if (tid < 32) scan_experts(cnt, base, E);
  __syncthreads();
  for (int e = tid; e < E; e += kPermThreads) counts[e] = cnt[e];
  for (int e = tid; e <= E; e += kPermThreads) offsets[e] = base[e];
  // rows that no pair takes (dropped pairs) read token 0, not what an earlier call left there
  for (int i = base[E] + tid; i < R; i += kPermThreads) row_token[i] = 0;
  for (int i0 = 0; i0 < R; i0 += kPermThreads)
    place_pairs(i0 + tid, expert_of(topk_ids, i0 + tid, R, E, nullptr), k, E, base, wcnt, row_token, pos);
}

// ---- multi-CTA variant: same result, two launches -------------------------------------------------
// A CTA per 1024 pairs counts them per expert; then every CTA adds up the counts of the chunks before its own
// (a few KB out of L2) and places its pairs. Chunks are ordered, so the placement stays ascending.
__global__ void __launch_bounds__(256)
permute_count_kernel(const int32_t* __restrict__ topk_ids, int R, int E, int32_t* __restrict__ chunk_cnt,
                     int32_t* __restrict__ err_flag, int32_t* __restrict__ pos, int32_t* __restrict__ zero_words, int zero_n) {
  __shared__ int cnt[kMaxExperts];
  wait_for_predecessor();
  for (int e = threadIdx.x; e < E; e += blockDim.x) cnt[e] = 0;
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < zero_n; i += blockDim.x) zero_words[i] = 0;
  __syncthreads();
  const int c0 = blockIdx.x * kPermThreads, c1 = min(R, c0 + kPermThreads);
  for (int i = c0 + threadIdx.x; i < c1; i += blockDim.x) {
    const int e = expert_of(topk_ids, i, R, E, err_flag);
    if (e >= 0) atomicAdd(&cnt[e], 1);
    else pos[i] = -1;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) chunk_cnt[(size_t)blockIdx.x * E + e] = cnt[e];
}

__global__ void __launch_bounds__(kPermThreads)
permute_place_kernel(const int32_t* __restrict__ topk_ids, int R, int k, int E, const int32_t* __restrict__ chunk_cnt,
                     int32_t* __restrict__ counts, int32_t* __restrict__ offsets, int32_t* __restrict__ row_token,
                     int32_t* __restrict__ pos, int tail_rows, int T) {
  __shared__ unsigned short wcnt[kPermWarps][kMaxExperts];
  __shared__ int tot[kMaxExperts], mine[kMaxExperts];
  __shared__ int base[kMaxExperts + 1];
  const int tid = threadIdx.x, n_chunks = gridDim.x;
  wait_for_predecessor();
  for (int i = blockIdx.x * kPermThreads + tid; i < tail_rows; i += n_chunks * kPermThreads) row_token[R + i] = i % T;
  for (int e = tid; e < E; e += kPermThreads) tot[e] = mine[e] = 0;
  __syncthreads();
  for (int x = tid; x < n_chunks * E; x += kPermThreads) {
    const int n = chunk_cnt[x], c = x / E;
    if (n > 0) {
      atomicAdd(&tot[x - c * E], n);
      if (c < (int)blockIdx.x) atomicAdd(&mine[x - c * E], n);
    }
  }
  __syncthreads();
  if (tid < 32) scan_experts(tot, base, E);
  __syncthreads();
  if (blockIdx.x == 0) {
    for (int e = tid; e < E; e += kPermThreads) counts[e] = tot[e];
    for (int e = tid; e <= E; e += kPermThreads) offsets[e] = base[e];
    for (int i = base[E] + tid; i < R; i += kPermThreads) row_token[i] = 0;  // rows that no pair takes
    __syncthreads();
  }
  if (tid < E) base[tid] += mine[tid];
  const int i = blockIdx.x * kPermThreads + tid;
  place_pairs(i, expert_of(topk_ids, i, R, E, nullptr), k, E, base, wcnt, row_token, pos);
}

// dst row r = src row index[r]; rows are row_vec 16-byte vectors long. A negative index (a pair the
// permutation dropped) yields a row of zeros.
__global__ void __launch_bounds__(256)
gather_rows_kernel(const uint4* __restrict__ src, const int32_t* __restrict__ index, int n_rows, int row_vec,
                   uint4* __restrict__ dst) {
  wait_for_predecessor();
  for (int r = blockIdx.x; r < n_rows; r += gridDim.x) {
    const int from = index[r];
    const uint4* s = src + (size_t)(from < 0 ? 0 : from) * row_vec;
    uint4* d = dst + (size_t)r * row_vec;
    for (int v = threadIdx.x; v < row_vec; v += blockDim.x) d[v] = from < 0 ? make_uint4(0, 0, 0, 0) : s[v];
  }
}

}  // namespace

cudaError_t launch_gather_rows(const void* src, const int32_t* index, int n_rows, size_t row_bytes, void* dst,
                               cudaStream_t s) {
  if (n_rows <= 0) return cudaSuccess;
  const int grid = n_rows < 1184 ? n_rows : 1184;  // 8 x 148 SMs
  return launch_behind(gather_rows_kernel, grid, 256, 0, s, (const uint4*)src, index, n_rows, (int)(row_bytes / 16), (uint4*)dst);
}

cudaError_t launch_permute(const int32_t* topk_ids, int R, int k, int E, int32_t* counts,
                           int32_t* offsets, int32_t* row_token, int32_t* pos, int32_t* err_flag,
                           int tail_rows, int T, cudaStream_t s, int32_t* scratch, size_t scratch_ints,
                           int32_t* zero_words, int zero_n) {
  if (zero_words == nullptr) zero_n = 0;
  // One CTA takes about 2 us per 1024 pairs.
  const int n_chunks = (R + kPermThreads - 1) / kPermThreads;
  if (n_chunks > 2 && scratch != nullptr && scratch_ints >= (size_t)n_chunks * E) {
    cudaError_t e = launch_behind(permute_count_kernel, n_chunks, 256, 0, s, topk_ids, R, E, scratch, err_flag, pos, zero_words, zero_n);
    if (e != cudaSuccess) return e;
    return launch_behind(permute_place_kernel, n_chunks, kPermThreads, 0, s, topk_ids, R, k, E, scratch, counts, offsets, row_token,
                         pos, tail_rows, T > 0 ? T : 1);
  }
  return launch_behind(permute_kernel, 1, kPermThreads, 0, s, topk_ids, R, k, E, counts, offsets, row_token, pos, err_flag, tail_rows,
                       T > 0 ? T : 1, zero_words, zero_n);
}

}  // namespace pm
