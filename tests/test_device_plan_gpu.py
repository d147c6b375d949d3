"""Launches planned on the device behind the router (resident experts and the shared expert, before the host has
read the row counts): experts with more rows than one chunk, absent experts, both kernels, against the float64
oracle; cache log exact. Every case says which kernel the call was planned for ("split", "tc", None = the host waits
for the counts) and the launch counters have to agree."""
import numpy as np
import pytest
import torch

from oracle import moe_math as om
from oracle import quant4 as oq
from oracle import srs_policy as sp
from promoe_b200 import _lib
from promoe_b200 import quant4 as pq
from promoe_b200.engine import ExpertCache
from tests.helpers import TinyModel, dev, dev_bf16

pytestmark = pytest.mark.gpu


def check(model, cache, T, rate, n_params, rtol, plan, steps=3):
    cache.enable_event_log(True)
    oc = sp.SequentialCache(model.L, model.E, model.k, cache_rate=rate, num_predict=0, num_per_expert_param=n_params)
    for x in model.hidden_stream(T, steps):
        for l in range(model.L):
            got = cache.forward(l, dev_bf16(x)).float().cpu().numpy()
            ref, _, _ = model.oracle_forward(l, x, report_experts=lambda u: np.asarray(oc.report_layer(l, u)))
            np.testing.assert_allclose(got, ref, rtol=rtol, atol=rtol * np.abs(ref).max() * 0.25)
            assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 8e-3
    assert cache.get("tc_error") == "0"
    for kind in ("split", "tc"):
        assert int(cache.get(f"planned_{kind}_launches")) == (steps * model.L if plan == kind else 0)
    assert cache.events() == oc.events
    cache.close()


# 9, 17 and 32 rows: either side of a chunk; 33 and 70: one to three 32-column granules; 610: experts of several
# token tiles (305 rows on average) and a ragged last granule
@pytest.mark.parametrize("T,plan", [(9, "split"), (17, "split"), (32, "split"), (33, "tc"), (70, "tc"), (610, "tc")])
@pytest.mark.parametrize("shared,rate", [(192, 1.0), (0, 1.0), (192, 0.5)])
def test_bf16_batches(lib, T, plan, shared, rate):
    model = TinyModel(seed=60 + T, L=2, E=4, H=192, I=64, k=2, shared_I=shared, shared_gate=shared > 0)
    check(model, model.make_cache(cache_rate=rate, num_predict_expert_per_layer=0), T, rate, 3, 2e-2, plan)


# chunks of 8 rows up to 8 rows per expert on average, then the host's plan, from 64 rows the tensor cores
@pytest.mark.parametrize("T,rate,plan", [(3, 1.0, "split"), (16, 1.0, "split"), (16, 0.5, "split"), (17, 1.0, None), (30, 1.0, None),
                                         (60, 1.0, None), (60, 0.5, None), (127, 0.5, None), (128, 1.0, "tc"), (610, 1.0, "tc"), (610, 0.5, "tc")])
def test_uint4_batches(lib, T, rate, plan):
    model = TinyModel(seed=90 + T, L=1, E=4, H=256, I=128, k=2, norm_topk=True, zipf_bias=False, gate_std=0.2)
    cache = ExpertCache(1, 4, num_expert_per_token=2, cache_rate=rate, num_predict_expert_per_layer=0)
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
    cache.set_layer_weights(0, dev_bf16(model.gate_w[0]), model.I, 2, True, quant4=True)
    check(model, cache, T, rate, 6, 3e-2, plan)


def q4_model_cache(model, rate):
    """A cache of the model's experts as uint4 (packed once and kept on the model)."""
    if not hasattr(model, "raw"):
        model.raw = [[[t for w in model.experts[l][e] for t in pq.quantize_pack(w)] for e in range(model.E)]
                     for l in range(model.L)]
    cache = ExpertCache(model.L, model.E, num_expert_per_token=model.k, cache_rate=rate, num_predict_expert_per_layer=0)
    cache.set_param_list(["w1.qweight", "w1.scale_zero", "w3.qweight", "w3.scale_zero", "w2.qweight", "w2.scale_zero"])
    for l in range(model.L):
        for e in range(model.E):
            cache.register_expert(l, e, model.raw[l][e])
    cache.pin_all()
    cache.build_slab()
    for l in range(model.L):
        cache.set_layer_weights(l, dev_bf16(model.gate_w[l]), model.I, model.k, model.norm_topk,
                                gate_bias=dev(model.gate_bias[l]), quant4=True)
    return cache


# experts that are found, that have to be copied, and that are copied one after another into too few lines: the launches
# differ, the numbers may not (T on either side of every line between two kernels)
@pytest.mark.parametrize("T", [20, 33, 48, 70, 200])
@pytest.mark.parametrize("kind", ["shared", "plain", "uint4"])
def test_outputs_do_not_depend_on_what_the_cache_held(lib, kind, T):
    model = TinyModel(seed=3 * T, L=1, E=8, H=1024, I=512, k=2, shared_I=512 if kind == "shared" else 0)
    xd = dev_bf16(model.hidden_stream(T, 1)[0])
    ys = []
    for rate in (1.0, 0.5, 0.25):
        cache = (q4_model_cache(model, rate) if kind == "uint4"
                 else model.make_cache(cache_rate=rate, num_predict_expert_per_layer=0))
        ys += [cache.forward(0, xd).clone() for _ in range(3)]
        assert cache.get("tc_error") == "0"
        cache.close()
    assert all(torch.equal(ys[0], y) for y in ys[1:])


# the chunks of the real rows against the kernel's table (264, uint4 128): fit; do not fit, with rows for the tensor cores and
# without; do not fit, uint4
@pytest.mark.parametrize("E,rows,bound,quant4", [(8, 20, 4, False), (64, 36, 8, False), (128, 30, 8, False), (100, 9, 1, True),
                                                 (8, 32, 32, False)])
def test_row_bound_below_the_truth_costs_no_row(lib, E, rows, bound, quant4):
    H = I = 128 if quant4 else 64
    model = TinyModel(seed=E + rows, L=1, E=E, H=H, I=I, k=1)
    n = min(E * rows, 8 * E if quant4 else E * rows)
    if quant4:
        cache = q4_model_cache(model, 1.0)
        mats = [[oq.dequantize(model.raw[0][e][2 * i], model.raw[0][e][2 * i + 1]) for i in range(3)] for e in range(E)]
    else:
        cache, mats = model.make_cache(cache_rate=1.0, num_predict_expert_per_layer=0), model.experts[0]
    cache.report_layer(0, list(range(E)))  # every expert is resident before the call
    for e in range(E):
        cache.expert_done(0, e)
    cache.layer_done(0)
    ids = (np.arange(n) // rows).astype(np.int32)
    np.random.default_rng(n).shuffle(ids)
    x = model.hidden_stream(n, 1)[0]
    xd, idd = dev_bf16(x), dev(ids)
    out = torch.full((n, H), float("nan"), dtype=torch.float32, device="cuda")
    for _ in range(2):
        _lib.call("pm_moe_forward_routed", cache.handle, 0, xd.data_ptr(), n, idd.data_ptr(), out.data_ptr(), bound, None, None,
                  0, 0, 0, 0, None)
        torch.cuda.synchronize()
    assert cache.get("tc_error") == "0"
    cache.close()
    got = out.cpu().numpy()
    for e in range(E):
        if (ids == e).any():
            ref = om.swiglu_mlp(x[ids == e], *mats[e], round_h_bf16=True)
            np.testing.assert_allclose(got[ids == e], ref, rtol=2e-2, atol=2e-2 * np.abs(ref).max() * 0.25)
