// Host side of the prefill (tcgen05) path: tensor-map encoding and tile planning for one segment.
#include <algorithm>
#include <cstring>

#include "runtime.hpp"

namespace pm {
namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// Innermost dimension k, zero fill. bf16: boxes 64 k (128 bytes) wide, 128-byte swizzle. Packed uint4
// (as bytes): boxes 128 k (64 bytes) wide, 64-byte swizzle, so that threads reading 16 bytes of
// neighbouring rows meet different banks.
int encode(CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
           const cuuint32_t* box, bool packed = false) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return fail(PM_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is not available");
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = fn(map, packed ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank,
                  const_cast<void*>(base), dims, strides_bytes, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  packed ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(PM_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult " + std::to_string((int)r));
  return PM_OK;
}

// Token rows: one map per box height.
int encode_rows(CUtensorMap (&maps)[4], const void* base, uint64_t k, uint64_t rows, uint64_t pitch_elems) {
  cuuint64_t dims[2] = {k, rows};
  cuuint64_t strides[1] = {pitch_elems * 2};
  for (int i = 0; i < 4; ++i) {
    cuuint32_t box[2] = {64, 16u << i};
    int rc = encode(&maps[i], base, 2, dims, strides, box);
    if (rc != PM_OK) return rc;
  }
  return PM_OK;
}

// Gate and up projections [inter, hidden] of `lines` experts `stride` bytes apart, as one map.
int encode_gate_up(CUtensorMap* map, int32_t* up_first, const unsigned char* gate, const unsigned char* up, uint64_t hidden,
                   uint64_t inter, uint64_t stride, uint64_t lines, bool packed = false) {
  *up_first = up < gate;
  const unsigned char* base = std::min(gate, up);
  const uint64_t apart = (uint64_t)(std::max(gate, up) - base);
  const uint64_t pitch = packed ? hidden / 2 : hidden * 2;
  cuuint64_t dims[5] = {packed ? hidden / 2 : hidden, 16, 2, inter / 16, lines};
  cuuint64_t strides[4] = {pitch, apart, pitch * 16, stride};
  cuuint32_t box[5] = {64, 16, 2, 4, 1};
  return encode(map, base, 5, dims, strides, box, packed);
}

int encode_down(CUtensorMap* map, const void* down, uint64_t hidden, uint64_t inter, uint64_t stride, uint64_t lines,
                bool packed = false) {
  cuuint64_t dims[3] = {packed ? inter / 2 : inter, hidden, lines};
  cuuint64_t strides[2] = {packed ? inter / 2 : inter * 2, stride};
  cuuint32_t box[3] = {64, 128, 1};
  return encode(map, down, 3, dims, strides, box, packed);
}

// Whether one map can span two matrices: its strides are positive and stay below 2^40 bytes. Allocators do place
// tensors of a program further apart than that.
bool one_map_spans(const void* a, const void* b) {
  const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b, apart = x > y ? x - y : y - x;
  return apart > 0 && apart < ((uintptr_t)1 << 40);
}

}  // namespace

bool tc_prefill_usable(const pm_ctx* c, const pm_layer_weights& w) {
  if (!c->tc_prefill || w.quant4 || encode_fn() == nullptr) return false;
  if (w.hidden % 64 != 0 || w.inter % 64 != 0 || w.shared_inter % 64 != 0) return false;
  return true;
}

bool tc_prefill_usable_q4(const pm_ctx* c, const pm_layer_weights& w) {
  if (!c->tc_prefill || !w.quant4 || encode_fn() == nullptr) return false;
  return w.hidden % 128 == 0 && w.inter % 128 == 0 && w.shared_inter % 64 == 0;
}

// Maps of the token rows, of the slab of expert lines and of the layer's shared expert. uint4 layers: the
// slab maps describe the packed matrices.
int tc_build_maps(pm_ctx* c, const pm_layer_weights& w, int rows_cap, TcMaps* m) {
  const uint64_t H = w.hidden, I = w.inter, Is = w.shared_inter, stride = c->line_stride, lines = c->n_lines;
  const bool packed = w.quant4 != 0;
  int rc = encode_rows(m->a_x, c->d_xperm, H, (uint64_t)rows_cap, H);
  if (rc != PM_OK) return rc;
  rc = encode_rows(m->a_h, c->d_hbuf, (uint64_t)c->ws_inter, (uint64_t)rows_cap, (uint64_t)c->ws_inter);
  if (rc != PM_OK) return rc;
  rc = encode_gate_up(&m->slab_gu, &m->slab_up_first, c->slab + c->param_offset[c->role_gate],
                      c->slab + c->param_offset[c->role_up], H, I, stride, lines, packed);
  if (rc != PM_OK) return rc;
  rc = encode_down(&m->slab_down, c->slab + c->param_offset[c->role_down], H, I, stride, lines, packed);
  if (rc != PM_OK) return rc;
  // never dereferenced where they stay as they are here: any valid map keeps the parameter well formed
  m->sh_gu = m->sh_up = m->slab_gu;
  m->sh_down = m->slab_down;
  m->sh_up_first = m->sh_split = 0;
  if (Is > 0) {
    m->sh_split = !one_map_spans(w.shared_w_gate, w.shared_w_up);
    if (m->sh_split) {
      const cuuint64_t dims[2] = {H, Is}, strides[1] = {H * 2};
      const cuuint32_t box[2] = {64, 16};
      rc = encode(&m->sh_gu, w.shared_w_gate, 2, dims, strides, box);
      if (rc == PM_OK) rc = encode(&m->sh_up, w.shared_w_up, 2, dims, strides, box);
    } else {  // one "line"; its stride is never used but has to be a valid one
      rc = encode_gate_up(&m->sh_gu, &m->sh_up_first, (const unsigned char*)w.shared_w_gate, (const unsigned char*)w.shared_w_up, H,
                          Is, H * 32, 1);
    }
    if (rc != PM_OK) return rc;
    rc = encode_down(&m->sh_down, w.shared_w_down, H, Is, Is * 2, 1);
    if (rc != PM_OK) return rc;
  }
  return PM_OK;
}

// Tiles of one group: token tiles of at most kTcMaxN rows times blocks of 128 gate/up rows or 256 down rows.
void tc_tile_count(const TcGroup& g, int hidden, int* gu, int* dn) {
  const int n = (g.row_count + kTcMaxN - 1) / kTcMaxN;
  *gu += n * ((g.inter + 127) / 128);
  *dn += n * ((hidden + 255) / 256);
}

}  // namespace pm
