// Shared declarations for the sm_100a kernels and the host runtime of the MoE hot path.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <string>
#include <vector>

#pragma GCC visibility push(default)
#include "../../include/promoe_b200.h"
#pragma GCC visibility pop

namespace pm {

// Records a message retrievable through pm_last_error(NULL) and returns `code`.
int fail(int code, const std::string& msg);
int fail_cuda(cudaError_t e, const char* what);
// PM_ERR_UNSUPPORTED (with a message naming `who`) while stream `s` is being captured into a graph.
int refuse_if_capturing(cudaStream_t s, const char* who);

#define PM_CUDA(expr)                                         \
  do {                                                        \
    cudaError_t pm_e_ = (expr);                               \
    if (pm_e_ != cudaSuccess) return pm::fail_cuda(pm_e_, #expr); \
  } while (0)

// One chunk of rows that share one set of FFN weights: a routed expert resolved
// to its cache slot, or a shared expert. Rows are positions in the permuted
// (expert-sorted) row order; a chunk never holds more than kMaxChunkRows rows.
struct GroupDesc {
  const void* w_gate;   // [inter, hidden] bf16, or packed uint4 [inter, hidden/2]
  const void* w_up;     // same layout as w_gate
  const void* w_down;   // [hidden, inter] bf16, or packed uint4 [hidden, inter/2]
  const void* q_gate;   // int4 only: per (row, 128-group) {scale, zero} fp16 pairs
  const void* q_up;
  const void* q_down;
  int32_t row_start;
  int32_t row_count;
  int32_t inter;
  int32_t tile_start_gu;  // first CTA tile of this chunk in the gate/up launch
  int32_t tile_start_dn;  // first CTA tile of this chunk in the down launch
  int32_t ld_down;        // row pitch of w_down in elements (0 = inter); larger when the chunk is one
                          // slice of a wider matrix's reduction dimension (fused decode kernel only)
};

constexpr int kTileRows = 64;       // weight rows per CTA tile of the staged kernel (4 warps x 16)
constexpr int kMaxChunkRows = 64;   // token rows per chunk (8 MMA n-tiles)
constexpr int kSplitMaxRows = 16;   // launches whose chunks all fit use the split-K decode kernel,
constexpr int kSplitTileGu = 16;    // whose tiles are 16 gate+up rows
constexpr int kSplitTileDn = 32;    // or 32 down rows
// Most rows of a bf16 group for which its layer call stays on the split-K kernel (as chunks of 16 rows). One group
// above it takes all groups of the call to the tensor cores, whose launch pair streams the weights of
// every group once; two kinds of launches after one another each leave SMs idle at their ends. Measured
// (FFN of one layer, mixed launches with the same line -> one kind): 64 tokens x top-8, experts of 1-40 rows
// (hidden 3584, inter 2560, shared 20480) 773 -> 716 us; 100 / 200 / 400 / 777 tokens x top-4 over 60 experts
// (2048 x 1408, shared 5632) 224 -> 204, 254 -> 228, 279 -> 247, 314 -> 269 us. With the line at 0, 32 tokens x
// top-6 over 64 experts lose: 155 us in chunks against 177 us. Above it, layer calls with a shared expert, chunks / tensor
// cores: 33, 48, 64 tokens over 64 experts of 2048 x 1408 180 / 195, 193 / 205, 210 / 205 us; over 64 of 3584 x 2560 (shared
// 20480) 749 / 664, 804 / 700, 920 / 700; over 8 of 4096 x 4096 183 / 172, 207 / 173, 230 / 174: the second reads
// of wide experts miss L2. (A line of its own for narrow ones, at 48, is not built.)
constexpr int kSplitChunkedMaxRows = 32;
// Fewest rows of a uint4 group that may run on the tensor cores. They take weights rounded to bf16 after
// dequantisation; the split-K tiles multiply the nibbles exactly and apply scale and zero to float32 sums
// (error of a layer call against 64 bits 2.4e-3 instead of 3.7e-3), and keep every group below this line.
constexpr int kQ4TcMinRows = 64;

// Launches of one layer call follow each other closely: with launch_behind a kernel may be scheduled while its
// predecessor in the stream drains (programmatic dependent launch). It has to call wait_for_predecessor before it
// touches what earlier kernels wrote; a predecessor lets it in early with let_successor_start, in every CTA, once all
// its own CTAs can be resident (a successor that waits may hold an SM). Walls of a pass, in turn on one GPU: one token
// 45.9 -> 43.6 us, two layers of 8 tokens with predictors 208.9 -> 191.4, 777 tokens 312 -> 299; routed rows gained no more than runs differ.
#ifdef __CUDACC__
// Opts a kernel in to all the dynamic shared memory a block can have beside its static part, once per device: the limit
// belongs to the function, so a launch that set it to its own need could take away what another thread's launch had just set.
struct SmemOptIn {
  std::atomic<char> done[64] = {};
};
template <class... P>
cudaError_t opt_in_smem(SmemOptIn& once, void (*kern)(P...)) {
  int dev = 0, most = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool known = dev >= 0 && dev < 64;
  if (known && once.done[dev].load(std::memory_order_acquire)) return cudaSuccess;
  cudaFuncAttributes attr{};
  if ((e = cudaFuncGetAttributes(&attr, kern)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)attr.sharedSizeBytes);
  if (e == cudaSuccess && known) once.done[dev].store(1, std::memory_order_release);
  return e;
}

__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_successor_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
cudaError_t launch_behind(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}
#endif

// Kernel launchers (defined in the .cu files). All take the caller's stream.
cudaError_t launch_gate_topk(const __nv_bfloat16* x, const __nv_bfloat16* w_gate, const float* bias,
                             const __nv_bfloat16* w_shared_gate, int T, int H, int E, int k,
                             int norm_topk, float routed_scale, const int32_t* expert_slot,
                             int32_t* topk_ids, float* topk_w, int32_t* topk_slot,
                             float* shared_scale, float* logits_out, cudaStream_t s);

// Router and permutation of a decode batch (at most 16 tokens) in one launch: launch_gate_topk followed by
// launch_permute on its ids. Usable when the token rows fit shared memory.
struct RouteArgs {
  const __nv_bfloat16 *x, *w_gate;
  const float* bias;
  const __nv_bfloat16* w_shared_gate;
  int32_t T, H, E, k, norm_topk;
  float routed_scale;
  const int32_t* expert_slot;
  int32_t* topk_ids;
  float* topk_w;
  int32_t* topk_slot;
  float* shared_scale;
  int32_t *counts, *offsets, *row_token, *pos, *err_flag;
  int32_t tail_rows, zero_n;
  int32_t* zero_words;
};
bool route_small_usable(int T, int H);
cudaError_t launch_route_small(const RouteArgs& a, cudaStream_t s);

// zero_words / zero_n: an int32 array the permutation also clears (the dependency counters of the
// fused FFN launch that follows on the same stream), or nullptr.
cudaError_t launch_permute(const int32_t* topk_ids, int R, int k, int E, int32_t* counts,
                           int32_t* offsets, int32_t* row_token, int32_t* pos, int32_t* err_flag,
                           int tail_rows, int T, cudaStream_t s, int32_t* scratch = nullptr,
                           size_t scratch_ints = 0, int32_t* zero_words = nullptr, int zero_n = 0);

// Geometry of one grouped FFN launch pair. The device blob it describes holds, 16-byte aligned
// and in this order: n_desc GroupDesc, tiles_gu int32 (chunk index of every gate/up CTA tile),
// tiles_dn int32 (same for the down launch), then n_desc + 1 int32 dependency counters that start
// at zero (the fused kernel counts the finished gate/up tiles per chunk and in total there) and one
// int32 error word.
struct FfnPlanInfo {
  int n_desc = 0, tiles_gu = 0, tiles_dn = 0, max_rows = 0, max_inter = 0;
  size_t off_tile_gu() const { return ((size_t)n_desc * sizeof(GroupDesc) + 15) / 16 * 16; }
  size_t off_tile_dn() const { return off_tile_gu() + ((size_t)tiles_gu * 4 + 15) / 16 * 16; }
  size_t off_counters() const { return off_tile_dn() + ((size_t)tiles_dn * 4 + 15) / 16 * 16; }
  size_t counter_bytes() const { return ((size_t)(n_desc + 2) * 4 + 15) / 16 * 16; }
  size_t blob_bytes() const { return off_counters() + counter_bytes(); }
};

// Splits caller groups into chunks of at most kMaxChunkRows rows, assigns CTA tile ranges and
// writes the blob into `blob` (host memory, `cap` bytes). Allocates nothing.
int plan_groups_into(const pm_ffn_group* groups, int n_groups, int hidden, unsigned char* blob, size_t cap,
                     FfnPlanInfo* info, int chunk_rows = kMaxChunkRows);
// Size pass of the same planner (blob == nullptr): fills `info` only.
int plan_groups_size(const pm_ffn_group* groups, int n_groups, int hidden, FfnPlanInfo* info,
                     int chunk_rows = kMaxChunkRows);

constexpr int kMaxSharedSlices = 8;
constexpr int kMaxFusedGroups = 256 + kMaxSharedSlices;  // groups of one fused launch
constexpr int kMaxFusedGroupsQ4 = 128;                    // same for uint4 experts (larger table records)
inline __host__ __device__ constexpr int fused_table_size(int quant4) { return quant4 ? kMaxFusedGroupsQ4 : kMaxFusedGroups; }

// What the fused kernel needs to describe, on the device, the shared expert and the routed experts
// a layer's slot table shows resident (no host round trip between the router and this launch).
// The shared expert is cut along its intermediate dimension into slices of `shared_slice` columns,
// each a group of its own with its own output rows (the combine adds them), so that every tile
// of the launch has about the same weight bytes.
// An expert (or slice) with more than chunk_rows rows becomes several chunks.
struct ResidentArgs {
  const int32_t* counts;      // [num_expert] routed rows per expert (permutation output)
  const int32_t* offsets;     // [num_expert + 1]
  const int32_t* slot_table;  // [num_expert] cache slot of each expert, -1 = absent
  const unsigned char* pool_base;  // first cache line of the layer's pool
  size_t line_stride;
  size_t off_gate, off_up, off_down;  // tensor offsets inside a line
  size_t off_qgate, off_qup, off_qdown;  // uint4 experts: scale / zero tensors
  const void *shared_w_gate, *shared_w_up, *shared_w_down;
  int32_t num_expert, inter, shared_inter, shared_slice;
  int32_t tokens, n_routed_rows;
  int32_t chunk_rows, quant4;
  int32_t max_rows;  // experts with more rows are left to the host's plan
};
// Rows per chunk of such a launch when an expert may have up to row_bound rows. bf16: the kernel variant for 8 rows
// or the one for 16. uint4: chunks of 8, the unpacking limits that kernel and its 16-row variant takes 1.6
// times as long per chunk, so an expert of 9-16 rows (unpacked twice) is the smaller cost.
inline int resident_chunk_rows(int row_bound, int quant4) { return quant4 || row_bound <= 8 ? 8 : 16; }
// Chunks of an expert with `rows` rows (0: left out).
inline __host__ __device__ int resident_chunks(const ResidentArgs& a, int rows) {
  return rows <= a.max_rows ? (rows + a.chunk_rows - 1) / a.chunk_rows : 0;
}
// Chunks of the shared expert: slices of its width, each over all tokens.
inline __host__ __device__ int resident_shared_chunks(const ResidentArgs& a) {
  return a.shared_inter > 0 ? (a.shared_inter + a.shared_slice - 1) / a.shared_slice * ((a.tokens + a.chunk_rows - 1) / a.chunk_rows) : 0;
}
// Most chunks such a launch can have if no expert has more than row_bound rows. A caller's bound may be wrong: a launch
// whose chunks do not fit the table does nothing, and the host, which counts them as the kernel does, plans it all.
inline int resident_max_chunks(const ResidentArgs& a, int row_bound) {
  const int most = row_bound < a.max_rows ? row_bound : a.max_rows;
  const int per = (most + a.chunk_rows - 1) / a.chunk_rows;
  const int routed = a.n_routed_rows / a.chunk_rows + a.num_expert;
  return (routed < per * a.num_expert ? routed : per * a.num_expert) + resident_shared_chunks(a);
}
// Width of one slice of a shared expert of width shared_inter beside routed experts of width inter.
inline int shared_slice_width(int inter, int shared_inter) {
  int w = inter > 0 ? inter : shared_inter;
  const int least = (shared_inter + kMaxSharedSlices - 1) / kMaxSharedSlices;
  if (w < least) w = least;
  w = (w + 31) / 32 * 32;
  return w < shared_inter ? w : shared_inter;
}
inline int shared_slice_count(int inter, int shared_inter) {
  if (shared_inter <= 0) return 0;
  const int w = shared_slice_width(inter, shared_inter);
  return (shared_inter + w - 1) / w;
}
// Launches the fused FFN for the shared expert (sliced) and every activated resident expert.
// counters: kMaxFusedGroups + 1 int32 (per chunk, then the launch total), zero at launch. err: a device word that receives a non-zero
// code if a bounded dependency wait gives up. Needs cooperative launch; does nothing where the chunks exceed the kernel's
// table (fused_table_size).
cudaError_t launch_resident_ffn(const ResidentArgs& a, int32_t* counters, int32_t* err,
                                const __nv_bfloat16* x, int hidden, const int32_t* row_token,
                                __nv_bfloat16* hbuf, int ld_h, float* yexp, cudaStream_t s);
bool resident_ffn_available(int chunk_rows, int quant4);

// Launches of at most kSplitMaxRows rows per chunk run as ONE cooperative kernel (gate/up tiles,
// then down tiles, a chunk's down tiles waiting on its gate/up tiles through the blob's counters),
// bf16 and uint4 alike (up to kMaxFusedGroups / kMaxFusedGroupsQ4 chunks); anything else runs as a gate/up and
// a down launch, and mid_event (optional) is recorded between the two. err (optional): device word
// that receives a code when a bounded wait of the fused kernel gives up (default: the blob's own
// error word).
cudaError_t launch_swiglu_ffn(const unsigned char* blob_dev, const FfnPlanInfo& info, int quant4,
                              const __nv_bfloat16* x, int H, const int32_t* row_token,
                              __nv_bfloat16* hbuf, int ld_h, float* yexp, cudaStream_t s,
                              cudaEvent_t mid_event = nullptr, int32_t* err = nullptr);
inline bool ffn_launch_is_fused(const FfnPlanInfo& info, int quant4) {
  return info.max_rows <= kSplitMaxRows && info.n_desc <= (quant4 ? kMaxFusedGroupsQ4 : kMaxFusedGroups);
}

cudaError_t launch_gather_rows(const void* src, const int32_t* index, int n_rows, size_t row_bytes, void* dst,
                               cudaStream_t s);

cudaError_t launch_combine(const float* yexp, const int32_t* pos, const float* topk_w, int T, int H,
                           int k, int R, int n_shared, const float* shared_scale,
                           __nv_bfloat16* y, cudaStream_t s);

// ---- tensor-core path (tcgen05) ------------------------------------------------------------------
// Tensor maps of one launch pair. Token rows (expert-sorted x, intermediate h): one map per box height
// 16, 32, 64, 128, so that a tile's rows arrive in as few boxes as possible (a box costs the copy engine
// about as much as 16 KB of data). Weights: routed experts through maps over the whole slab whose last
// coordinate is the cache line, the layer's shared expert through maps of its own. The gate/up maps
// see both matrices as (k, row in block of 16, matrix, block, line), so that one box of 4 blocks brings
// 64 gate and 64 up rows, alternating in blocks of 16; the matrix with the lower address comes first. The
// matrices of a shared expert are the caller's and may lie further apart than a map's stride reaches: then sh_split is set,
// sh_gu and sh_up are 2-D maps of one matrix each, and a box brings 16 rows.
struct TcMaps {
  CUtensorMap a_x[4], a_h[4], slab_gu, slab_down, sh_gu, sh_up, sh_down;
  int32_t slab_up_first, sh_up_first, sh_split;
};
struct TcGroup {
  int32_t row_start, row_count, inter;
  int32_t line;  // global cache line of the expert, -1 = the shared expert
};
// The groups of a launch pair as the device knows them behind the router: the shared expert (if any) and every
// activated expert the layer's slot table shows resident. Experts with fewer than min_rows rows are left to the host's plan.
struct TcPlan {
  const int32_t *counts, *offsets, *slot_table;
  int32_t num_expert, first_line;  // first_line: global cache line of slot 0
  int32_t inter, shared_inter, tokens, n_routed_rows, min_rows;
};
constexpr int kTcMaxN = 256;       // token rows per tile
constexpr int kMaxTcGroups = 264;  // groups of one launch pair (every expert and the shared one)
struct TcLaunch {
  const TcMaps* maps;
  const TcGroup* groups_dev;   // nullptr: the groups of `plan`
  TcPlan plan;
  int n_groups, max_rows;      // groups, rows of the largest (with a plan: bounds)
  int tiles_gu, tiles_dn;      // tiles of the two launches (tc_tile_count), which bound their grids
  int hidden, ld_h;
  __nv_bfloat16* hbuf;
  float* yexp;
  int32_t* err_dev;
  // uint4 experts (scale_base non-null; the slab maps then describe the packed matrices): {scale, zero} pairs
  // of cache line l at scale_base + l * scale_stride + the projection's offset
  const unsigned char* scale_base = nullptr;
  size_t scale_stride = 0, scale_gate = 0, scale_up = 0, scale_down = 0;
};
cudaError_t launch_prefill_ffn(const TcLaunch& a, cudaStream_t s, cudaEvent_t mid_event);

// out[r] = index of the r-th best of scores[0 .. width) (descending, ties to the lower index), r < n.
cudaError_t launch_rank_topn(const float* scores, int width, int n, int32_t* out, cudaStream_t s);

cudaError_t launch_predictor_mlp(const __nv_bfloat16* x, int B, int H, const __nv_bfloat16* w1,
                                 const float* b1, int D, const __nv_bfloat16* w2, const float* b2,
                                 int E, float* hidden_scratch, float* scores, cudaStream_t s);

// The same followed by launch_rank_topn on its scores, in one launch less. E at most 256.
cudaError_t launch_predictor_ranked(const __nv_bfloat16* x, int B, int H, const __nv_bfloat16* w1, const float* b1, int D,
                                    const __nv_bfloat16* w2, const float* b2, int E, float* hidden_scratch, float* scores,
                                    int n, int32_t* out, cudaStream_t s);

}  // namespace pm
