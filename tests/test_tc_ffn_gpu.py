"""The tensor-core grouped FFN (csrc/ffn_tcgen05.cu) at the edges of its tiles: rows per expert around the
32-column granule and the 256-row tile, widths that are not multiples of the weight tiles, both orders of
the gate and up matrices in memory. Exact row counts come through pm_moe_forward_routed; the oracle is
the float64 SwiGLU on the same bf16 inputs."""
import numpy as np
import pytest
import torch

from oracle import moe_math as om
from oracle import quant4 as oq
from promoe_b200 import _lib
from promoe_b200 import quant4 as pq
from promoe_b200.engine import ExpertCache
from tests.helpers import TinyModel, bf16_weights, dev_bf16

pytestmark = pytest.mark.gpu


def run_routed(lib, H, I, counts, names=("gate_proj.weight", "up_proj.weight", "down_proj.weight"), seed=5):
    E = len(counts)
    model = TinyModel(seed=seed, L=1, E=E, H=H, I=I, k=1)
    cache = ExpertCache(1, E, num_expert_per_token=1, cache_rate=1.0, num_predict_expert_per_layer=0)
    cache.set_param_list(list(names))
    kind = {"gate_proj.weight": 0, "up_proj.weight": 1, "down_proj.weight": 2}
    for e in range(E):
        cache.register_expert(0, e, [om.to_bf16_bits(model.experts[0][e][kind[n]]) for n in names])
    cache.pin_all()
    cache.build_slab()
    cache.set_layer_weights(0, None, I, 1, False, 1.0, hidden=H)
    rng = np.random.default_rng(seed)
    ids = np.repeat(np.arange(E, dtype=np.int32), counts)
    ids = np.concatenate([ids, np.full(3, -1, np.int32)])  # padding rows
    rng.shuffle(ids)
    n = len(ids)
    x = om.bf16_round(rng.standard_normal((n, H)).astype(np.float32))
    xd, idd = dev_bf16(x), torch.from_numpy(ids).cuda()
    out = torch.full((n, H), float("nan"), dtype=torch.float32, device="cuda")
    for _ in range(2):  # the second call meets a workspace that holds the first one's rows
        _lib.call("pm_moe_forward_routed", cache.handle, 0, xd.data_ptr(), n, idd.data_ptr(), out.data_ptr(), 0, None, None,
                  0, 0, 0, 0, None)
        torch.cuda.synchronize()
    assert cache.get("tc_error") == "0"
    launches = int(cache.get("tc_launches"))
    cache.close()
    got = out.cpu().numpy()
    ref = np.zeros((n, H))
    for e in range(E):
        if counts[e]:
            at = ids == e
            ref[at] = om.swiglu_mlp(x[at], *model.experts[0][e], round_h_bf16=True)
    # both sides round the intermediate row to bf16 from sums in another order: a flipped rounding moves
    # one of I products by 2^-8, far below these bounds
    np.testing.assert_allclose(got, ref, rtol=2e-2, atol=2e-2 * np.abs(ref).max() * 0.25)
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 5e-3
    return launches


@pytest.mark.parametrize("H,I,counts", [
    (64, 64, [33, 0, 64, 65]),            # one k-step, less than one weight tile
    (320, 192, [255, 256, 257, 1]),       # either side of a full token tile; ragged weight tiles
    (1024, 448, [513, 40, 96, 7]),        # three token tiles, a K loop longer than the stage ring
    (256, 128, [700, 0, 0, 0]),
    (512, 256, [33] * 80),                # more tiles than CTA pairs, all of them small
])
def test_tile_edges(lib, H, I, counts):
    assert run_routed(lib, H, I, counts) > 0


# up to 64 rows, less than three chunks per group and few weights: the split-K tiles; a row more on one expert, or three
# chunks per group: the tensor cores
@pytest.mark.parametrize("counts,tc", [([64, 5, 16, 1], False), ([33, 32, 0, 0], False), ([65, 5, 16, 1], True), ([33, 33], True)])
def test_few_weights_stay_in_chunks(lib, counts, tc):
    assert (run_routed(lib, 256, 192, counts) > 0) == tc


def test_up_matrix_first_in_memory(lib):
    assert run_routed(lib, 256, 192, [70, 130, 33], names=("up_proj.weight", "down_proj.weight", "gate_proj.weight")) > 0


@pytest.mark.parametrize("H,I,counts", [
    (128, 128, [64, 0, 70]),              # one k-step
    (640, 384, [129, 256, 257, 3]),       # either side of a full token tile, ragged weight tiles
    (1024, 1152, [600, 64]),              # K loops longer than the rings, two and three token tiles
    (256, 256, [65] * 24),                # more tiles than CTA pairs
])
def test_uint4_tile_edges(lib, H, I, counts):
    rng = np.random.default_rng(H + I)
    E, deq = len(counts), []
    cache = ExpertCache(1, E, num_expert_per_token=1, cache_rate=1.0, num_predict_expert_per_layer=0)
    cache.set_param_list(["w1.qweight", "w1.scale_zero", "w3.qweight", "w3.scale_zero", "w2.qweight", "w2.scale_zero"])
    for e in range(E):
        raw, mats = [], []
        for shape in ((I, H), (I, H), (H, I)):
            packed, sz = pq.quantize_pack(bf16_weights(rng, shape))
            raw += [packed, sz]
            mats.append(oq.dequantize(packed, sz))
        deq.append(mats)
        cache.register_expert(0, e, raw)
    cache.pin_all()
    cache.build_slab()
    cache.set_layer_weights(0, None, I, 1, False, 1.0, hidden=H, quant4=True)
    ids = np.repeat(np.arange(E, dtype=np.int32), counts)
    rng.shuffle(ids)
    n = len(ids)
    x = om.bf16_round(rng.standard_normal((n, H)).astype(np.float32))
    xd, idd = dev_bf16(x), torch.from_numpy(ids).cuda()
    out = torch.full((n, H), float("nan"), dtype=torch.float32, device="cuda")
    for _ in range(2):
        _lib.call("pm_moe_forward_routed", cache.handle, 0, xd.data_ptr(), n, idd.data_ptr(), out.data_ptr(), 0, None, None,
                  0, 0, 0, 0, None)
        torch.cuda.synchronize()
    assert cache.get("tc_error") == "0" and int(cache.get("q4_expanded")) > 0
    cache.close()
    got, ref = out.cpu().numpy(), np.zeros((n, H))
    for e in range(E):
        if counts[e]:
            ref[ids == e] = om.swiglu_mlp(x[ids == e], *deq[e], round_h_bf16=True)
    # weights rounded to bf16 after dequantisation: 2^-9 per product, independent, on top of the bf16 path's error
    np.testing.assert_allclose(got, ref, rtol=3e-2, atol=3e-2 * np.abs(ref).max() * 0.25)
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 8e-3


def test_uint4_layer_with_bf16_shared_expert(lib):
    """The shared expert of a uint4 layer is bf16: decode rows and prompt rows both reach it."""
    model = TinyModel(seed=8, L=1, E=4, H=256, I=128, k=2, shared_I=192)
    rng = np.random.default_rng(3)
    cache = ExpertCache(1, 4, num_expert_per_token=2, cache_rate=1.0, num_predict_expert_per_layer=0)
    cache.set_param_list(["w1.qweight", "w1.scale_zero", "w3.qweight", "w3.scale_zero", "w2.qweight", "w2.scale_zero"])
    for e in range(4):
        raw, mats = [], []
        for w in model.experts[0][e]:
            packed, sz = pq.quantize_pack(w)
            raw += [packed, sz]
            mats.append(oq.dequantize(packed, sz))
        model.experts[0][e] = tuple(mats)
        cache.register_expert(0, e, raw)
    cache.pin_all()
    cache.build_slab()
    cache.set_layer_weights(0, dev_bf16(model.gate_w[0]), model.I, 2, False,
                            gate_bias=None if model.gate_bias is None else torch.from_numpy(model.gate_bias[0]).cuda(),
                            shared=[dev_bf16(w) for w in model.shared[0]], quant4=True)
    for T in (5, 40, 300):
        x = om.bf16_round(rng.standard_normal((T, model.H)).astype(np.float32))
        y = cache.forward(0, dev_bf16(x)).float().cpu().numpy()
        ref, _, _ = model.oracle_forward(0, x)
        assert np.linalg.norm(y - ref) / np.linalg.norm(ref) < 8e-3
    cache.close()


@pytest.mark.parametrize("rows", [40, 20])  # the tensor cores; the split-K tiles
def test_silu_of_large_negative_gates(lib, rows):
    """The quotient -g / (1 + e^g) just above g = 87 is a normal float32 (some 1e-36) that a large up value brings
    back into range; an approximate division returns 0 for denominators above 2^126."""
    H = I = 64
    rng = np.random.default_rng(rows)
    wg, wu = np.zeros((I, H), np.float32), np.zeros((I, H), np.float32)
    wg[:, 0] = rng.choice([-87.5, -88.0, -88.5, -3.0, 2.0], size=I)
    wu[:, 0] = np.where(wg[:, 0] < -87, np.float32(2.0) ** 100, np.float32(2.0) ** -20)
    wd = bf16_weights(rng, (H, I))
    cache = ExpertCache(1, 1, num_expert_per_token=1, cache_rate=1.0, num_predict_expert_per_layer=0)
    cache.set_param_list(["gate_proj.weight", "up_proj.weight", "down_proj.weight"])
    cache.register_expert(0, 0, [om.to_bf16_bits(m) for m in (wg, wu, wd)])
    cache.pin_all()
    cache.build_slab()
    cache.set_layer_weights(0, None, I, 1, False, 1.0, hidden=H)
    x = np.zeros((rows, H), np.float32)
    x[:, 0] = 1.0
    xd, idd = dev_bf16(x), torch.zeros(rows, dtype=torch.int32, device="cuda")
    out = torch.empty((rows, H), dtype=torch.float32, device="cuda")
    _lib.call("pm_moe_forward_routed", cache.handle, 0, xd.data_ptr(), rows, idd.data_ptr(), out.data_ptr(), 0, None, None,
              0, 0, 0, 0, None)
    torch.cuda.synchronize()
    assert (int(cache.get("tc_launches")) > 0) == (rows > 32)
    cache.close()
    ref = om.swiglu_mlp(x, wg, wu, wd, round_h_bf16=True)
    assert np.abs(ref).max() > 1e-8
    # __expf is off by 2 ulp + |x| * 2^-22 in its exponent (2e-5 here), the row is rounded to bf16
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=2e-2, atol=2e-2 * np.abs(ref).max() * 0.25)


class FarPair:
    """Two device buffers 2^41 bytes apart: one address range with memory mapped at its two ends."""

    def __init__(self, nbytes):
        from cuda.bindings import driver as cu
        self.cu, dev_id = cu, torch.cuda.current_device()
        torch.zeros(1, device="cuda")
        prop = cu.CUmemAllocationProp()
        prop.type = cu.CUmemAllocationType.CU_MEM_ALLOCATION_TYPE_PINNED
        prop.location.type = cu.CUmemLocationType.CU_MEM_LOCATION_TYPE_DEVICE
        prop.location.id = dev_id
        gran = self.ok(cu.cuMemGetAllocationGranularity(prop, cu.CUmemAllocationGranularity_flags.CU_MEM_ALLOC_GRANULARITY_MINIMUM))
        self.size = -(-nbytes // gran) * gran
        self.total = (1 << 41) + self.size
        self.base = int(self.ok(cu.cuMemAddressReserve(self.total, gran, 0, 0)))
        acc = cu.CUmemAccessDesc()
        acc.location = prop.location
        acc.flags = cu.CUmemAccess_flags.CU_MEM_ACCESS_FLAGS_PROT_READWRITE
        self.at, self.handles = [self.base, self.base + (1 << 41)], []
        for a in self.at:
            h = self.ok(cu.cuMemCreate(self.size, prop, 0))
            self.ok(cu.cuMemMap(a, self.size, 0, h, 0))
            self.ok(cu.cuMemSetAccess(a, self.size, [acc], 1))
            self.handles.append(h)

    def ok(self, r):
        assert int(r[0]) == 0, r[0]
        return r[1] if len(r) > 1 else None

    def tensor(self, i, like):
        """A bf16 tensor over buffer i with the values of `like`."""
        class Raw:
            __cuda_array_interface__ = {"shape": tuple(like.shape), "typestr": "<i2", "data": (self.at[i], False), "version": 3}
        t = torch.as_tensor(Raw(), device="cuda").view(torch.bfloat16)
        t.copy_(like)
        return t

    def free(self):
        torch.cuda.synchronize()
        for a, h in zip(self.at, self.handles):
            self.ok(self.cu.cuMemUnmap(a, self.size))
            self.ok(self.cu.cuMemRelease(h))
        self.ok(self.cu.cuMemAddressFree(self.base, self.total))


@pytest.mark.parametrize("where", ["far", "far, up first", "same"])
@pytest.mark.parametrize("H,Is,T", [(64, 64, 70), (320, 448, 300)])
def test_shared_matrices_that_one_map_cannot_span(lib, where, H, Is, T):
    """The gate and up matrices of a shared expert further apart than a tensor map's stride reaches (or one and the
    same): still on the tensor cores, bit-equal to matrices that lie together."""
    model = TinyModel(seed=T + Is, L=1, E=4, H=H, I=64, k=2, shared_I=Is)
    wg, wu, wd = (dev_bf16(m) for m in model.shared[0])
    if where == "same":
        wu = wg.clone()
    x, ys = dev_bf16(model.hidden_stream(T, 1)[0]), []
    far = FarPair(wg.numel() * 2)
    for split in (False, True):
        if not split:
            shared = [wg, wu, wd]
        elif where == "same":
            shared = [wg, wg, wd]
        else:
            order = (1, 0) if where == "far, up first" else (0, 1)
            shared = [far.tensor(order[0], wg), far.tensor(order[1], wu), wd]
        cache = model.make_cache(cache_rate=1.0, num_predict_expert_per_layer=0)
        cache.set_layer_weights(0, dev_bf16(model.gate_w[0]), model.I, 2, False, gate_bias=torch.from_numpy(model.gate_bias[0]).cuda(),
                                shared=shared)
        ys.append(cache.forward(0, x).clone())
        assert cache.get("tc_error") == "0" and int(cache.get("tc_launches")) > 0
        cache.close()
    far.free()
    assert torch.equal(ys[0], ys[1])
    model.shared[0] = (model.shared[0][0], model.shared[0][0] if where == "same" else model.shared[0][1], model.shared[0][2])
    ref, _, _ = model.oracle_forward(0, x.float().cpu().numpy())
    assert np.linalg.norm(ys[1].float().cpu().numpy() - ref) / np.linalg.norm(ref) < 8e-3
