// K3b: grouped SwiGLU expert FFN on the 5th-generation tensor cores, for experts with more rows than the
// split-K decode tiles take (swiglu_ffn.cu). A pair of CTAs (cta_group::2) computes one tile: 256 weight
// rows as the M operand (128 gate + the same 128 up rows, or 256 down rows) times up to 256 token rows
// as the N operand. Weights on M and tokens on N because N can be any multiple of 32: an expert's rows
// are cut into equal tiles of at most 256, so little work goes to padding, and an expert with 20 rows
// streams its weights once against a 32-column tile.
//
// What bounds it: many rows per expert, the operands' way from L2 through the ring (a k-step of 64 moves 32 KB per
// CTA for 4.2 Mflop, half of each token tile comes from the pair's other CTA): the tensor pipe is busy 61 % (gate/up) and
// 54 % (down) of the time, L2 at 39 % and DRAM at 33-42 % of their peaks. Few rows, HBM (six stages keep about
// 100 KB of weight loads in flight per SM). Measured on 8192 tokens x top-6 over 64 experts (hidden 2048, inter
// 1408) + a shared expert of 2816: gate/up 622-630 us = 1200-1216 TFLOP/s, down 364-368 us = 1026-1038 TFLOP/s (747 and
// 471 us with one-CTA tiles of 128 token rows and a 2-stage ring). In a timing experiment the gate/up main loop took
// 621 us without its epilogue (660 with it on that box), 509 us with the token loads left out too.
//
// Persistent: one pair per two SMs walks the tiles pair, pair + n_pairs, ... Warp 0 loads (TMA, 128-byte
// swizzle, 6-stage mbarrier ring), one thread of the pair's first CTA issues the MMAs, and eight warps per
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
// uint4 experts (Q4): the packed matrices are read straight from the cache lines. TMA brings packed rows into a
// ring of their own, eight warps expand each weight once per 256 token rows to bf16 ((q - zero) * scale in
// float32, rounded once) and write it where TMA would have put it, behind a proxy fence. 8 experts of 4096 x
// 14336, 512 tokens x top-2: gate/up 375 us, down 210 us (writing a bf16 copy of every expert first and reading it back
// took 813 us plus 630 us for the products). What bounds this: with up to 64 rows per expert gate/up took 340 us, 282 us
// without the expansion's arithmetic (22 instructions per 8 weights); the larger part is the packed weights'
// way from HBM, through the two 8 KB slots that three stages for 256 columns leave. The rounding of the weights is why
// groups of fewer than kQ4TcMinRows rows do not come here.
//
// It replaces, for batches with many rows per expert, the per-expert torch linears the
// reference runs in its Python expert loop (src/sparse_llm_cache/utils/hooks.py:187-198).
//
// Every mbarrier wait is bounded; on a give-up the kernel records a code in *err, stops all roles of
// the CTA (the pair's other CTA runs into its own limit), frees its tensor memory and returns.
#include <algorithm>

#include "pm_common.cuh"
#include "sm100_ptx.cuh"

namespace pm {

namespace {

using namespace sm100;

constexpr int kEpiWarps = 8;      // two per quadrant of the accumulator rows
constexpr int kDequantWarps = 8;  // uint4 experts: two threads per weight row of a stage
template <bool Q4>
constexpr int tc_threads() { return (4 + kEpiWarps + (Q4 ? kDequantWarps : 0)) * 32; }
// k per stage in swizzle atoms of 64 (128 bytes of bf16): one, or a whole quantisation group for uint4
template <bool Q4>
constexpr int tc_atoms() { return Q4 ? 2 : 1; }
constexpr int kAtomBytes = 128 * 128;       // one CTA's 128 weight rows of an atom
constexpr int kRawBytes = 128 * 64;         // the same rows' packed weights of a uint4 stage
constexpr int kMaxStages = 12, kMaxRaw = 8;
constexpr uint32_t kTmemCols = 512;         // two accumulators of 256 columns

struct TcSlot {  // one group in shared memory
  int32_t row_start, rows, line, inter;
  int32_t width, n_tiles;  // columns per token tile, token tiles
  int32_t first_tile;
};

struct TcShared {
  uint64_t full[kMaxStages], empty[kMaxStages], raw_full[kMaxRaw], raw_empty[kMaxRaw], acc_full[2], acc_empty[2];
  uint32_t sz[kMaxRaw][128];  // {scale, zero} of the packed rows in the raw ring
  uint32_t tmem_base;
  volatile int abort;
  int n_groups, n_tiles;
  TcSlot slot[kMaxTcGroups];
};

// Ring geometry of a launch: the token part of a stage is as large as the launch's widest tile needs, the
// number of stages follows.
struct TcRing {
  int32_t stage_bytes, n_stages, n_raw;
  size_t smem_bytes() const {
    return 1024 /*alignment slack*/ + (size_t)stage_bytes * n_stages + (size_t)kRawBytes * n_raw + sizeof(TcShared);
  }
};
template <bool Q4>
TcRing ring_for(int max_rows) {
  // a group of more than 256 rows may have tiles of any width up to 256
  const int half = max_rows > kTcMaxN ? kTcMaxN / 2 : (max_rows + 31) / 32 * 16;
  TcRing r;
  r.stage_bytes = tc_atoms<Q4>() * (kAtomBytes + half * 128);
  const int room = 232448 - 1024 - (int)sizeof(TcShared);
  if (Q4) {
    // two stages cover the hand-over between the expanding warps and the MMAs, a third the token rows' way from
    // L2; the rest (two slots at least, which the expanding warps need) holds packed weights on their way from HBM
    r.n_stages = 3;
    r.n_raw = std::min(kMaxRaw, (room - r.n_stages * r.stage_bytes) / kRawBytes);
  } else {
    r.n_stages = std::min(kMaxStages, room / r.stage_bytes);
    r.n_raw = 0;
  }
  return r;
}

// Where the {scale, zero} pairs of the cache lines are: base + line * stride + offset.
struct TcScales {
  const unsigned char* base;
  size_t stride, gate, up, down;
  uint32_t exponent;  // 0x4B000000, see nibble_at
};

// Position in a ring of n slots with the parity of the current turn.
struct RingPos {
  int slot = 0;
  uint32_t turn = 0;
  __device__ __forceinline__ void next(int n) {
    if (++slot == n) {
      slot = 0;
      ++turn;
    }
  }
};

// Group table: token tiles of equal width (a multiple of 32, at most 256) and the tile ranges.
template <bool GATEUP>
__device__ __forceinline__ void build_table(TcShared& sh, const TcGroup* __restrict__ groups, const TcPlan& plan, int n_groups,
                                            int hidden) {
  for (int i = threadIdx.x; i < n_groups; i += blockDim.x) {
    TcGroup g;
    if (groups != nullptr) {
      g = groups[i];
    } else {  // group 0 is the shared expert where there is one, then the experts in order, those left out with no rows
      const int e = i - (plan.shared_inter > 0 ? 1 : 0);
      if (e < 0) {
        g = TcGroup{plan.n_routed_rows, plan.tokens, plan.shared_inter, -1};
      } else {
        const int slot = plan.slot_table[e], rows = plan.counts[e];
        g = TcGroup{plan.offsets[e], slot >= 0 && rows >= plan.min_rows ? rows : 0, plan.inter, plan.first_line + slot};
      }
    }
    TcSlot t;
    t.row_start = g.row_start;
    t.rows = g.row_count;
    t.line = g.line;
    t.inter = g.inter;
    t.n_tiles = (g.row_count + kTcMaxN - 1) / kTcMaxN;
    t.width = t.n_tiles > 0 ? ((g.row_count + t.n_tiles - 1) / t.n_tiles + 31) / 32 * 32 : 0;
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

__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t pack_u32x2(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
// Two nibbles of a word, left in place under the exponent of 2^23 (the float is 2^23 + q * 2^position, exact),
// become bf16 weights: the subtraction of 2^23 is exact, the fused multiply-add rounds
// q * scale - zero * scale once (zero * scale is a product of two fp16 values, exact in float32).
__device__ __forceinline__ uint32_t q4_weights(uint32_t lo_bits, uint32_t hi_bits, uint64_t scale, uint64_t minus_zs) {
  const uint64_t magic = pack_u32x2(0xCB000000u, 0xCB000000u);  // (-2^23, -2^23)
  uint64_t q, w;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(q) : "l"(pack_u32x2(lo_bits, hi_bits)), "l"(magic));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(w) : "l"(q), "l"(scale), "l"(minus_zs));
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(w));
  const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&p);
}
// `exponent` is 0x4B000000 (2^23), held in a register: a logic instruction takes one immediate only, and with
// both constants known the compiler spends two.
template <int POS>
__device__ __forceinline__ uint32_t nibble_at(uint32_t word, uint32_t exponent) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(word), "n"(0xF << POS), "r"(exponent));  // (word & mask) | exponent
  return r;
}

template <bool GATEUP, bool Q4>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(tc_threads<Q4>(), 1)
prefill_ffn_kernel(const __grid_constant__ TcMaps maps, const __grid_constant__ TcScales scales, const TcRing ring,
                   const TcGroup* __restrict__ groups, const TcPlan plan, int n_groups, int hidden,
                   __nv_bfloat16* __restrict__ hbuf, int ld_h, float* __restrict__ yexp, int32_t* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  // the same offset in both CTAs of the pair: the MMA addresses both through one descriptor
  unsigned char* stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* raw = stages + (size_t)ring.n_stages * ring.stage_bytes;
  TcShared& sh = *reinterpret_cast<TcShared*>(raw + (size_t)ring.n_raw * kRawBytes);
  constexpr int kAtoms = tc_atoms<Q4>(), kStageK = 64 * kAtoms, kWBytes = kAtoms * kAtomBytes;
  constexpr int kFirstDequant = 4 + kEpiWarps;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int n_stages = ring.n_stages;

  // The down pass may start while the gate/up pass drains; it waits where it first needs its results (the producer
  // of its token rows). What both read besides is complete before the gate/up pass lets it in.
  if (GATEUP) wait_for_predecessor();
  let_successor_start();
  if (threadIdx.x == 0) {
    for (int s = 0; s < n_stages; ++s) {
      mbar_init(&sh.full[s], 1 + (Q4 ? 2 * kDequantWarps : 0));
      mbar_init(&sh.empty[s], 1);
    }
    for (int r = 0; r < ring.n_raw; ++r) {
      mbar_init(&sh.raw_full[r], 1 + 32);  // the TMA thread, and the 32 lanes that bring the scales
      mbar_init(&sh.raw_empty[r], kDequantWarps);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&sh.acc_full[a], 1);
      mbar_init(&sh.acc_empty[a], 2 * kEpiWarps);  // the epilogue warps of both CTAs
    }
    sh.abort = 0;
    fence_barrier_init();
  }
  if (warp == 2) tmem_alloc(&sh.tmem_base, kTmemCols);
  build_table<GATEUP>(sh, groups, plan, n_groups, hidden);
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem_base = sh.tmem_base;
  const int n_tiles = sh.n_tiles;

  if (warp == 0 && lane == 0) {
    // ---- producer: this CTA's half of the weight rows (bf16 experts) and of the token rows ---------
    if (!GATEUP) wait_for_predecessor();
    TileAt t;
    RingPos at;
    int steps = 0;
    bool ok = true;
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
      t.seek(sh, tile);
      const TcSlot& g = sh.slot[t.gi];
      const bool shared_expert = g.line < 0;
      const int line = shared_expert ? 0 : g.line;
      const CUtensorMap* map_w = GATEUP ? (shared_expert ? &maps.sh_gu : &maps.slab_gu) : (shared_expert ? &maps.sh_down : &maps.slab_down);
      const CUtensorMap* map_x = GATEUP ? maps.a_x : maps.a_h;
      const int k_tiles = (GATEUP ? hidden : g.inter) / kStageK;
      const int half = t.width / 2;
      const int x_row = g.row_start + t.n0 + (int)rank * half;
      const uint32_t bytes = 2u * (uint32_t)((Q4 ? 0 : kWBytes) + kAtoms * half * 128);
      for (int kt = 0; kt < k_tiles; ++kt, ++steps, at.next(n_stages)) {
        if (at.turn > 0 && !mbar_wait(&sh.empty[at.slot], (at.turn - 1) & 1, &sh.abort)) {
          ok = false;
          break;
        }
        if (rank == 0) mbar_arrive_expect_tx(&sh.full[at.slot], bytes);
        const uint32_t bar = map_to_rank(smem_u32(&sh.full[at.slot]), 0);
        unsigned char* dst = stages + (size_t)at.slot * ring.stage_bytes;
        if (!Q4) {
          if (GATEUP && shared_expert && maps.sh_split) {
#pragma unroll 1
            for (int b = 0; b < 8; ++b)  // 16 gate rows, the 16 up rows, the next 16 gate rows, ...
              tma_load_2d(dst + b * 2048, b & 1 ? &maps.sh_up : &maps.sh_gu, bar, kt * 64, t.m * 128 + (int)rank * 64 + (b >> 1) * 16);
          } else if (GATEUP) tma_load_5d(dst, map_w, bar, kt * 64, 0, 0, t.m * 8 + (int)rank * 4, line);
          else tma_load_3d(dst, map_w, bar, kt * 64, t.m * 256 + (int)rank * 128, line);
        }
        dst += kWBytes;
#pragma unroll
        for (int a = 0; a < kAtoms; ++a) {
          int row = x_row;
#pragma unroll
          for (int i = 3; i >= 0; --i)  // half is a multiple of 16: one box per set bit
            if (half & (16 << i)) {
              tma_load_2d(dst, map_x + i, bar, kt * kStageK + a * 64, row);
              dst += (16 << i) * 128;
              row += 16 << i;
            }
        }
      }
    }
    // the last arrivals on this CTA's barriers must have landed before its shared memory goes away
    for (int k = max(0, steps - n_stages); k < steps && ok; ++k)
      ok = mbar_wait(&sh.empty[k % n_stages], (k / n_stages) & 1, &sh.abort);
    if (!ok) {
      atomicExch(err, 1);
      sh.abort = 1;
    }
  } else if (Q4 && warp == 2 && lane == 0) {
    // ---- packed weights of this CTA's rows: HBM -> raw ring -----------------------------------------
    TileAt t;
    RingPos at;
    bool ok = true;
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
      t.seek(sh, tile);
      const TcSlot& g = sh.slot[t.gi];
      const int k_tiles = (GATEUP ? hidden : g.inter) / kStageK;
      for (int kt = 0; kt < k_tiles; ++kt, at.next(ring.n_raw)) {
        if (at.turn > 0 && !mbar_wait(&sh.raw_empty[at.slot], (at.turn - 1) & 1, &sh.abort)) {
          ok = false;
          break;
        }
        mbar_arrive_expect_tx(&sh.raw_full[at.slot], kRawBytes);
        const uint32_t bar = map_to_rank(smem_u32(&sh.raw_full[at.slot]), rank);
        unsigned char* dst = raw + (size_t)at.slot * kRawBytes;
        if (GATEUP) tma_load_5d(dst, &maps.slab_gu, bar, kt * 64, 0, 0, t.m * 8 + (int)rank * 4, g.line);
        else tma_load_3d(dst, &maps.slab_down, bar, kt * 64, t.m * 256 + (int)rank * 128, g.line);
      }
    }
    if (!ok) {
      atomicExch(err, 5);
      sh.abort = 1;
    }
  } else if (Q4 && warp == 3) {
    // ---- scales of the same rows, asynchronously and by a warp of its own: a load in flight in the
    // expanding warps would hold up the fence behind their shared-memory writes -------------------------
    TileAt t;
    RingPos at;
    bool ok = true;
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
      t.seek(sh, tile);
      const TcSlot& g = sh.slot[t.gi];
      const int k_tiles = (GATEUP ? hidden : g.inter) / kStageK;
      const unsigned char* line = scales.base + (size_t)g.line * scales.stride;
      const uint32_t* src[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int row = j * 32 + lane;
        if (GATEUP) {
          const bool up = (lane >= 16) != (maps.slab_up_first != 0);
          const int r = min(t.m * 128 + (int)rank * 64 + j * 16 + (lane & 15), g.inter - 1);
          src[j] = reinterpret_cast<const uint32_t*>(line + (up ? scales.up : scales.gate)) + (size_t)r * k_tiles;
        } else {
          const int r = min(t.m * 256 + (int)rank * 128 + row, hidden - 1);
          src[j] = reinterpret_cast<const uint32_t*>(line + scales.down) + (size_t)r * k_tiles;
        }
      }
      for (int kt = 0; kt < k_tiles; ++kt, at.next(ring.n_raw)) {
        const bool free = at.turn == 0 || mbar_wait(&sh.raw_empty[at.slot], (at.turn - 1) & 1, &sh.abort);
        if (!__all_sync(0xffffffffu, free)) {
          ok = false;
          break;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) cp_async_4(smem_u32(&sh.sz[at.slot][j * 32 + lane]), src[j] + kt);
        cp_async_arrive(&sh.raw_full[at.slot]);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!ok && lane == 0) {
      atomicExch(err, 5);
      sh.abort = 1;
    }
  } else if (Q4 && warp >= kFirstDequant) {
    // ---- expand: a thread turns half of one row's quantisation group (a stage) into bf16, written where TMA
    // would have put them (128-byte swizzle). The packed words of the next stage are in registers and its
    // barriers polled before a stage's writes are fenced, so that only the arithmetic is left on the chain from
    // stage to stage.
    constexpr int kChunks = 16 / kDequantWarps;  // 16-byte pieces (32 weights) of packed words per thread
    const int idx = threadIdx.x - kFirstDequant * 32;
    const int row = idx & 127, part = idx >> 7;
    const uint32_t ex = scales.exponent;
    uint32_t src0[kChunks], dst0[kChunks];
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      const int q = part * kChunks + c;  // quarter of the quantisation group
      // 64-byte swizzle of the packed tile: 16-byte piece q of row r sits at q ^ ((r >> 1) & 3)
      src0[c] = smem_u32(raw) + row * 64 + ((q ^ ((row >> 1) & 3)) << 4);
      dst0[c] = (smem_u32(stages) + (q >> 1) * kAtomBytes + row * 128) | ((((q & 1) * 4) ^ (row & 7)) << 4);
    }
    const uint32_t sz0 = smem_u32(&sh.sz[0][row]), empty0 = smem_u32(&sh.empty[0]), raw_full0 = smem_u32(&sh.raw_full[0]);
    const uint32_t raw_empty0 = smem_u32(&sh.raw_empty[0]), full0 = map_to_rank(smem_u32(&sh.full[0]), 0);
    int steps = 0;
    {
      TileAt t;
      for (int tile = pair; tile < n_tiles; tile += n_pairs) {
        t.seek(sh, tile);
        steps += (GATEUP ? hidden : sh.slot[t.gi].inter) / kStageK;
      }
    }
    RingPos at, rat;
    bool ok = true;
    uint4 w4[kChunks];
    uint32_t sz = 0;
    if (steps > 0) {
      ok = __all_sync(0xffffffffu, mbar_wait(raw_full0, 0, &sh.abort));
#pragma unroll
      for (int c = 0; c < kChunks; ++c) w4[c] = lds128(src0[c]);
      sz = lds32(sz0);
    }
    for (int step = 0; step < steps && ok; ++step) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&sz));  // x = scale, y = zero
      const float s4 = f.x * 0.0625f, s8 = f.x * 0.00390625f, s12 = f.x * 0.000244140625f, s16 = f.x * 0.0000152587890625f;
      const uint64_t c0 = pack_f32x2(f.x, s16), c1 = pack_f32x2(s4, s8), c2 = pack_f32x2(s8, s12), c3 = pack_f32x2(s12, s16);
      const float mzs = -f.x * f.y;
      const uint64_t mz = pack_f32x2(mzs, mzs);
#pragma unroll
      for (int n = 0; n < 4 * kChunks; ++n) {
        const uint32_t w = (&w4[n / 4].x)[n % 4], dst = dst0[n / 4] + at.slot * ring.stage_bytes;
        const uint32_t v = w >> 12;  // nibbles 5, 6, 7 at 8, 12, 16
        sts128(dst ^ ((n % 4) << 4), q4_weights(nibble_at<0>(w, ex), nibble_at<16>(w, ex), c0, mz),
               q4_weights(nibble_at<4>(w, ex), nibble_at<8>(v, ex), c1, mz),
               q4_weights(nibble_at<8>(w, ex), nibble_at<12>(v, ex), c2, mz),
               q4_weights(nibble_at<12>(w, ex), nibble_at<16>(v, ex), c3, mz));
      }
      const uint32_t done_raw = raw_empty0 + rat.slot * 8, done_stage = full0 + at.slot * 8;
      at.next(n_stages);
      rat.next(ring.n_raw);
      if (step + 1 < steps) {
        const uint32_t rf = raw_full0 + rat.slot * 8;
        bool got;
        if (at.turn > 0) got = mbar_wait2(rf, rat.turn & 1, empty0 + at.slot * 8, (at.turn - 1) & 1, &sh.abort);
        else got = mbar_wait(rf, rat.turn & 1, &sh.abort);  // the first turn finds every stage free
        ok = __all_sync(0xffffffffu, got);
#pragma unroll
        for (int c = 0; c < kChunks; ++c) w4[c] = lds128(src0[c] + rat.slot * kRawBytes);
        sz = lds32(sz0 + rat.slot * 512);
      }
      fence_proxy_async();  // the tensor core reads these writes through the async proxy
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(done_raw);
        mbar_arrive_cluster(done_stage);
      }
    }
    if (!ok && lane == 0) {
      atomicExch(err, 6);
      sh.abort = 1;
    }
  } else if (warp == 1 && lane == 0 && rank == 0) {
    // ---- MMA issuer for both CTAs ------------------------------------------------------------------
    TileAt t;
    RingPos at;
    int it = 0;
    bool ok = true;
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, ++it) {
      t.seek(sh, tile);
      const int k_tiles = (GATEUP ? hidden : sh.slot[t.gi].inter) / kStageK;
      const int acc = it & 1;
      if (it >= 2 && !mbar_wait(&sh.acc_empty[acc], ((it >> 1) - 1) & 1, &sh.abort)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t idesc = umma_idesc_bf16(256, t.width);
      const uint32_t d = tmem_base + (uint32_t)acc * 256;
      const uint32_t x_atom = (uint32_t)t.width * 64;  // bytes of this CTA's token rows of an atom
      for (int kt = 0; kt < k_tiles; ++kt, at.next(n_stages)) {
        if (!mbar_wait(&sh.full[at.slot], at.turn & 1, &sh.abort)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(stages + (size_t)at.slot * ring.stage_bytes);
#pragma unroll
        for (int k = 0; k < kStageK / 16; ++k)  // UMMA K = 16 bf16 = 32 bytes inside the swizzled row
          umma_bf16(d, umma_desc_k_sw128(a_addr + (k / 4) * kAtomBytes + (k % 4) * 32),
                    umma_desc_k_sw128(a_addr + kWBytes + (k / 4) * x_atom + (k % 4) * 32), idesc,
                    (kt > 0 || k > 0) ? 1u : 0u);
        umma_commit_pair(&sh.empty[at.slot]);  // the stage may be refilled once these MMAs have read it
      }
      if (ok) umma_commit_pair(&sh.acc_full[acc]);
    }
    if (!ok) {
      atomicExch(err, 2);
      sh.abort = 1;
    }
  } else if (warp >= 4 && warp < kFirstDequant) {
    // ---- epilogue: warp w owns accumulator rows 32w .. 32w+31 of this CTA; two warps of one quadrant share
    // the columns ----------------------------------------------------------------------------------------
    const int w = warp & 3, first = ((warp - 4) >> 2) * 32, stride = kEpiWarps * 8;
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
      for (int c0 = first; c0 < t.cols; c0 += stride) {
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
            const float h = gv / (1.f + __expf(-gv)) * uv;  // a full division: __fdividef gives 0 for denominators above 2^126
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
int resident_pairs() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (dev >= 0 && dev < 64 && cached[dev] > 0) return cached[dev];
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  // the attribute is per device: a process that drives several GPUs opts in on each of them
  for (auto kern : {prefill_ffn_kernel<true, false>, prefill_ffn_kernel<false, false>, prefill_ffn_kernel<true, true>,
                    prefill_ffn_kernel<false, true>})
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448) != cudaSuccess) return 0;
  if (dev >= 0 && dev < 64) cached[dev] = sms / 2;
  return sms / 2;
}

template <bool Q4>
cudaError_t launch_pair(const TcLaunch& a, cudaStream_t s, cudaEvent_t mid_event) {
  const int pairs = resident_pairs();
  if (pairs <= 0) return cudaErrorNotSupported;
  const TcRing ring = ring_for<Q4>(a.max_rows);
  const TcScales sc{a.scale_base, a.scale_stride, a.scale_gate, a.scale_up, a.scale_down, 0x4B000000u};
  const size_t smem = ring.smem_bytes();
  cudaError_t e = launch_behind(prefill_ffn_kernel<true, Q4>, 2 * std::min(pairs, a.tiles_gu), tc_threads<Q4>(), smem, s, *a.maps,
                                sc, ring, a.groups_dev, a.plan, a.n_groups, a.hidden, a.hbuf, a.ld_h, a.yexp, a.err_dev);
  if (e != cudaSuccess) return e;
  if (mid_event != nullptr) {
    e = cudaEventRecord(mid_event, s);
    if (e != cudaSuccess) return e;
  }
  return launch_behind(prefill_ffn_kernel<false, Q4>, 2 * std::min(pairs, a.tiles_dn), tc_threads<Q4>(), smem, s, *a.maps, sc,
                       ring, a.groups_dev, a.plan, a.n_groups, a.hidden, a.hbuf, a.ld_h, a.yexp, a.err_dev);
}

}  // namespace

cudaError_t launch_prefill_ffn(const TcLaunch& a, cudaStream_t s, cudaEvent_t mid_event) {
  if (a.n_groups <= 0) return cudaSuccess;
  if (a.n_groups > kMaxTcGroups) return cudaErrorInvalidValue;
  return a.scale_base != nullptr ? launch_pair<true>(a, s, mid_event) : launch_pair<false>(a, s, mid_event);
}

}  // namespace pm
