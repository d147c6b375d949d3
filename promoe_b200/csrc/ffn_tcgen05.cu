// K3b: grouped SwiGLU expert FFN on the 5th-generation tensor cores, for experts with more rows than the
// split-K decode tiles take (swiglu_ffn.cu). A pair of CTAs (cta_group::2) computes one tile: 256 weight
// rows as the M operand (128 gate + the same 128 up rows, or 256 down rows) times up to 256 token rows
// as the N operand. Weights on M and tokens on N because N can be any multiple of 32: an expert's rows
// are cut into equal tiles of at most 256, so little work goes to padding, and an expert with 20 rows
// streams its weights once against a 32-column tile.
//
// What bounds it: many rows per expert, the operands' way from L2 to the SMs (a k-step of 64 moves 32 KB per
// CTA for 4.2 Mflop, half of each token tile comes from the pair's other CTA); few rows, HBM (six
// stages keep about 100 KB of weight loads in flight per SM). Measured on 8192 tokens x top-6 over 64
// experts (hidden 2048, inter 1408) + a shared expert of 2816: gate/up 660 us = 1146 TFLOP/s, down 378 us =
// 1000 TFLOP/s (747 and 471 us with one-CTA tiles of 128 token rows and a 2-stage ring). Without its
// epilogue the gate/up main loop takes 621 us, with the token loads left out too 509 us: the operand
// traffic, about 10 TB/s out of L2, is what is left.
//
// Persistent: one pair per two SMs walks the tiles pair, pair + n_pairs, ... Warp 0 loads (TMA, 128-byte
// swizzle, 6-stage mbarrier ring), one thread of the pair's first CTA issues the MMAs, and four warps per
// CTA drain the accumulators, which are double-buffered in tensor memory (2 x 256 columns) so that an
// epilogue runs under the next tile's MMAs. Gate and up rows alternate in blocks of 16, so that a warp's
// 32 accumulator rows are 16 gate rows and the 16 up rows that go with them: one shuffle per two columns
// brings a pair together.
//
// Rows are the expert-sorted token rows (gathered once per layer call), so an expert's rows are
// contiguous; a tile may run past the expert's last row into its neighbour's rows or past the
// end of the buffer (TMA zero fill): those columns are computed and never stored. Expert weights
// are addressed by cache line through ONE 3-D tensor map per projection over the whole slab
// (k, weight row, line); the shared expert has 2-D maps of its own. No multicast loads are used.
//
// It replaces, for batches with many rows per expert, the per-expert torch linears the
// reference runs in its Python expert loop (src/sparse_llm_cache/utils/hooks.py:187-198).
//
// Every mbarrier wait is bounded; on a give-up the kernel records a code in *err, stops all roles of
// the pair, frees its tensor memory and returns.
#include <algorithm>

#include "pm_common.cuh"
#include "sm100_ptx.cuh"

namespace pm {

namespace {

using namespace sm100;

constexpr int kEpiWarps = 8;                    // two per quadrant of the accumulator rows
constexpr int kTcThreads = (4 + kEpiWarps) * 32;
constexpr int kTcStages = 6;
constexpr int kBK = 64;                         // k per stage (128 bytes of bf16)
constexpr int kWBytes = 128 * kBK * 2;          // one CTA's weight rows of a stage
constexpr int kXBytes = (kTcMaxN / 2) * kBK * 2;  // one CTA's token rows of a stage (at most)
constexpr int kStageBytes = kWBytes + kXBytes;
constexpr uint32_t kTmemCols = 512;             // two accumulators of 256 columns

struct TcSlot {  // one group in shared memory
  int32_t row_start, rows, line, inter;
  int32_t width, n_tiles;  // columns per token tile, token tiles
  int32_t first_tile;
};

struct TcShared {
  uint64_t full[kTcStages], empty[kTcStages], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  volatile int abort;
  int n_groups, n_tiles;
  TcSlot slot[kMaxTcGroups];
};

constexpr size_t tc_smem_bytes() { return 1024 /*alignment slack*/ + (size_t)kTcStages * kStageBytes + sizeof(TcShared); }

// Group table: token tiles of equal width (a multiple of 32, at most 256) and the tile ranges.
template <bool GATEUP>
__device__ __forceinline__ void build_table(TcShared& sh, const TcGroup* __restrict__ groups, int n_groups, int hidden) {
  for (int i = threadIdx.x; i < n_groups; i += kTcThreads) {
    const TcGroup g = groups[i];
    TcSlot t;
    t.row_start = g.row_start;
    t.rows = g.row_count;
    t.line = g.line;
    t.inter = g.inter;
    t.n_tiles = (g.row_count + kTcMaxN - 1) / kTcMaxN;
    t.width = ((g.row_count + t.n_tiles - 1) / t.n_tiles + 31) / 32 * 32;
    const int m_tiles = GATEUP ? (g.inter + 127) / 128 : (hidden + 255) / 256;
    t.first_tile = t.n_tiles * m_tiles;  // a count; the scan below turns it into a position
    sh.slot[i] = t;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int run = 0;
    for (int c = 0; c < n_groups; c += 32) {
      const int i = c + threadIdx.x;
      const int n = i < n_groups ? sh.slot[i].first_tile : 0;
      int incl = n;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, d);
        if ((int)threadIdx.x >= d) incl += v;
      }
      if (i < n_groups) sh.slot[i].first_tile = run + incl - n;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (threadIdx.x == 0) {
      sh.n_groups = n_groups;
      sh.n_tiles = run;
    }
  }
  __syncthreads();
}

struct TileAt {
  int gi = 0;
  int m, n0, cols, width;  // weight tile, first token row inside the group, valid columns, MMA columns
  // Tiles only move forward. Token tiles of one weight tile are neighbours, so they share its weights in L2.
  __device__ __forceinline__ void seek(const TcShared& sh, int tile) {
    while (gi + 1 < sh.n_groups && sh.slot[gi + 1].first_tile <= tile) ++gi;
    const TcSlot& s = sh.slot[gi];
    const int local = tile - s.first_tile;
    m = local / s.n_tiles;
    width = s.width;
    n0 = (local - m * s.n_tiles) * s.width;
    cols = min(width, s.rows - n0);
  }
};

template <bool GATEUP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kTcThreads, 1)
prefill_ffn_kernel(const __grid_constant__ TcMaps maps, const TcGroup* __restrict__ groups, int n_groups, int hidden,
                   __nv_bfloat16* __restrict__ hbuf, int ld_h, float* __restrict__ yexp, int32_t* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  // the same offset in both CTAs of the pair: the MMA addresses both through one descriptor
  unsigned char* stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  TcShared& sh = *reinterpret_cast<TcShared*>(stages + (size_t)kTcStages * kStageBytes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kTcStages; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&sh.acc_full[a], 1);
      mbar_init(&sh.acc_empty[a], 2 * kEpiWarps);  // the epilogue warps of both CTAs
    }
    sh.abort = 0;
    fence_barrier_init();
  }
  if (warp == 2) tmem_alloc(&sh.tmem_base, kTmemCols);
  build_table<GATEUP>(sh, groups, n_groups, hidden);
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem_base = sh.tmem_base;
  const int n_tiles = sh.n_tiles;

  if (warp == 0 && lane == 0) {
    // ---- producer: this CTA's half of the weight rows and of the token rows ------------------------
    TileAt t;
    int step = 0;
    bool ok = true;
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
      t.seek(sh, tile);
      const TcSlot& g = sh.slot[t.gi];
      const bool shared_expert = g.line < 0;
      const int line = shared_expert ? 0 : g.line;
      const CUtensorMap* map_w = GATEUP ? (shared_expert ? &maps.sh_gu : &maps.slab_gu) : (shared_expert ? &maps.sh_down : &maps.slab_down);
      const CUtensorMap* map_x = GATEUP ? maps.a_x : maps.a_h;
      const int k_tiles = (GATEUP ? hidden : g.inter) / kBK;
      const int half = t.width / 2;
      const int x_row = g.row_start + t.n0 + (int)rank * half;
      const uint32_t bytes = 2u * (uint32_t)(kWBytes + half * kBK * 2);
      for (int kt = 0; kt < k_tiles; ++kt, ++step) {
        const int s = step % kTcStages;
        if (step >= kTcStages && !mbar_wait(&sh.empty[s], ((step / kTcStages) - 1) & 1, &sh.abort)) {
          ok = false;
          break;
        }
        if (rank == 0) mbar_arrive_expect_tx(&sh.full[s], bytes);
        const uint32_t bar = map_to_rank(smem_u32(&sh.full[s]), 0);
        unsigned char* dst = stages + (size_t)s * kStageBytes;
        if (GATEUP) tma_load_5d(dst, map_w, bar, kt * kBK, 0, 0, t.m * 8 + (int)rank * 4, line);
        else tma_load_3d(dst, map_w, bar, kt * kBK, t.m * 256 + (int)rank * 128, line);
        dst += kWBytes;
        int row = x_row;
#pragma unroll
        for (int i = 3; i >= 0; --i)  // half is a multiple of 16: one box per set bit
          if (half & (16 << i)) {
            tma_load_2d(dst, map_x + i, bar, kt * kBK, row);
            dst += (16 << i) * kBK * 2;
            row += 16 << i;
          }
      }
    }
    // the last arrivals on this CTA's barriers must have landed before its shared memory goes away
    for (int k = max(0, step - kTcStages); k < step && ok; ++k)
      ok = mbar_wait(&sh.empty[k % kTcStages], (k / kTcStages) & 1, &sh.abort);
    if (!ok) {
      atomicExch(err, 1);
      sh.abort = 1;
    }
  } else if (warp == 1 && lane == 0 && rank == 0) {
    // ---- MMA issuer for both CTAs ------------------------------------------------------------------
    TileAt t;
    int step = 0, it = 0;
    bool ok = true;
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, ++it) {
      t.seek(sh, tile);
      const int k_tiles = (GATEUP ? hidden : sh.slot[t.gi].inter) / kBK;
      const int acc = it & 1;
      if (it >= 2 && !mbar_wait(&sh.acc_empty[acc], ((it >> 1) - 1) & 1, &sh.abort)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t idesc = umma_idesc_bf16(256, t.width);
      const uint32_t d = tmem_base + (uint32_t)acc * 256;
      for (int kt = 0; kt < k_tiles; ++kt, ++step) {
        const int s = step % kTcStages;
        if (!mbar_wait(&sh.full[s], (step / kTcStages) & 1, &sh.abort)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(stages + (size_t)s * kStageBytes);
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k)  // UMMA K = 16 bf16 = 32 bytes inside the swizzled row
          umma_bf16(d, umma_desc_k_sw128(a_addr + k * 32), umma_desc_k_sw128(a_addr + kWBytes + k * 32), idesc,
                    (kt > 0 || k > 0) ? 1u : 0u);
        umma_commit_pair(&sh.empty[s]);  // the stage may be refilled once these MMAs have read it
      }
      if (ok) umma_commit_pair(&sh.acc_full[acc]);
    }
    if (!ok) {
      atomicExch(err, 2);
      sh.abort = 1;
    }
  } else if (warp >= 4) {
    // ---- epilogue: warp w owns accumulator rows 32w .. 32w+31 of this CTA, and every second block of 32
    // columns ----------------------------------------------------------------------------------------
    const int w = warp & 3, first = ((warp - 4) >> 2) * 32;
    TileAt t;
    int it = 0;
    bool ok = true;
    for (int tile = pair; tile < n_tiles; tile += n_pairs, ++it) {
      t.seek(sh, tile);
      const TcSlot& g = sh.slot[t.gi];
      const int acc = it & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(&sh.acc_full[acc], (it >> 1) & 1, &sh.abort))) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t taddr = tmem_base + (uint32_t)acc * 256 + ((uint32_t)(32 * w) << 16);
      const size_t row0 = (size_t)(g.row_start + t.n0);
#pragma unroll 1
      for (int c0 = first; c0 < t.cols; c0 += 64) {
        uint32_t v[32];
        tmem_ld32(taddr + c0, v);
        tmem_ld_wait();
        if (GATEUP) {
          // 16 lanes hold gate rows, the other 16 the matching up rows: of two neighbouring columns the
          // lower half of the warp finishes the first, the upper half the second
          const bool upper = lane >= 16, up_first = g.line < 0 ? maps.sh_up_first : maps.slab_up_first;
          const int i = t.m * 128 + (int)rank * 64 + w * 16 + (lane & 15);
          __nv_bfloat16* dst = hbuf + (row0 + c0 + (upper ? 1 : 0)) * ld_h + i;
          const int left = (i < g.inter) ? t.cols - c0 - (upper ? 1 : 0) : 0;
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            const uint32_t other = __shfl_xor_sync(0xffffffffu, upper ? v[c] : v[c + 1], 16);
            const uint32_t lo = upper ? other : v[c], hi = upper ? v[c + 1] : other;
            const float gv = __uint_as_float(up_first ? hi : lo), uv = __uint_as_float(up_first ? lo : hi);
            const float h = __fdividef(gv, 1.f + __expf(-gv)) * uv;
            if (c < left) dst[(size_t)c * ld_h] = __float2bfloat16_rn(h);
          }
        } else {
          const int n = t.m * 256 + (int)rank * 128 + w * 32 + lane;
          float* dst = yexp + (row0 + c0) * hidden + n;
          const int left = n < hidden ? t.cols - c0 : 0;
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (c < left) dst[(size_t)c * hidden] = __uint_as_float(v[c]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&sh.acc_empty[acc]), 0));
    }
    if (!ok && lane == 0) {
      atomicExch(err, 3);
      sh.abort = 1;
    }
  }
  __syncwarp();
  __syncthreads();
  // give loads that are still in flight time to land before the shared memory is released
  if (sh.abort)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  if (warp == 2) tmem_dealloc(tmem_base, kTmemCols);
}

// Pairs that fit the device at once (0 on error).
int resident_pairs(int dev) {
  static int cached[64] = {};
  if (dev >= 0 && dev < 64 && cached[dev] > 0) return cached[dev];
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  // the attribute is per device: a process that drives several GPUs opts in on each of them
  for (auto kern : {prefill_ffn_kernel<true>, prefill_ffn_kernel<false>})
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc_smem_bytes()) != cudaSuccess) return 0;
  if (dev >= 0 && dev < 64) cached[dev] = sms / 2;
  return sms / 2;
}

}  // namespace

cudaError_t launch_prefill_ffn(const TcMaps& maps, const TcGroup* groups_dev, int n_groups, int tiles_gu, int tiles_dn,
                               int hidden, __nv_bfloat16* hbuf, int ld_h, float* yexp, int32_t* err_dev, cudaStream_t s,
                               cudaEvent_t mid_event) {
  if (n_groups <= 0) return cudaSuccess;
  if (n_groups > kMaxTcGroups) return cudaErrorInvalidValue;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const int pairs = resident_pairs(dev);
  if (pairs <= 0) return cudaErrorNotSupported;
  prefill_ffn_kernel<true><<<2 * std::min(pairs, tiles_gu), kTcThreads, tc_smem_bytes(), s>>>(maps, groups_dev, n_groups, hidden,
                                                                                   hbuf, ld_h, yexp, err_dev);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (mid_event != nullptr) {
    e = cudaEventRecord(mid_event, s);
    if (e != cudaSuccess) return e;
  }
  prefill_ffn_kernel<false><<<2 * std::min(pairs, tiles_dn), kTcThreads, tc_smem_bytes(), s>>>(maps, groups_dev, n_groups, hidden,
                                                                                    hbuf, ld_h, yexp, err_dev);
  return cudaGetLastError();
}

}  // namespace pm
