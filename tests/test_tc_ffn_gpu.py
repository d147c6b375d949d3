"""The tensor-core grouped FFN (csrc/ffn_tcgen05.cu) at the edges of its tiles: rows per expert around the
32-column granule and the 256-row tile, widths that are not multiples of the weight tiles, both orders of
the gate and up matrices in memory. Exact row counts come through pm_moe_forward_routed; the oracle is
the float64 SwiGLU on the same bf16 inputs."""
import numpy as np
import pytest
import torch

from oracle import moe_math as om
from promoe_b200 import _lib
from promoe_b200.engine import ExpertCache
from tests.helpers import TinyModel, dev_bf16

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


def test_up_matrix_first_in_memory(lib):
    assert run_routed(lib, 256, 192, [70, 130, 33], names=("up_proj.weight", "down_proj.weight", "gate_proj.weight")) > 0
