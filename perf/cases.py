"""Performance cases of the expert-cached MoE layer: what is timed, and on which sizes.

A case is one configuration of the layer call that a model makes for every MoE layer and every step
(`ExpertCache.forward`, its host-buffer form `ExpertCache.forward_host`, and the row-routed form
`pm_moe_forward_routed` that an expert-parallel owner calls). Weights, router, shared expert and the
expert cache are what a program keeps between calls; the token rows are the input of a pass.

`kind` of a case:
  layer   one layer call with every expert resident (T tokens: decode for small T, a prompt for large T)
  host    the same from and to pinned host buffers
  stack   `steps` decode steps of `L` layers, optionally with the next-layer predictors and with fewer
          cache lines than experts (cache_rate), so that missing experts are copied from the host
  routed  the owner side of an expert-parallel layer: rows that other ranks routed, with padding rows
"""
from __future__ import annotations

import ctypes
import math

import torch

from promoe_b200 import _lib
from promoe_b200.engine import ExpertCache

STD = 0.02     # weights ~ N(0, 0.02)
PRED_D = 512   # hidden width of the predictor MLPs


def _case(kind, T, H, I, E, k, shared=0, shared_gate=False, norm=False, q4=False, L=1, steps=1, rate=1.0,
          predict=0, world=1):
    return dict(kind=kind, T=T, H=H, I=I, E=E, k=k, shared=shared, shared_gate=shared_gate, norm=norm, q4=q4, L=L,
                steps=steps, rate=rate, predict=predict, world=world)


# Shapes of the repository's configurations.
DSMOE = dict(H=2048, I=1408, E=64, k=6, shared=2816)                         # DeepSeek-MoE-16B / V2-Lite
QWEN = dict(H=2048, I=1408, E=60, k=4, shared=5632, shared_gate=True)        # Qwen1.5-MoE-A2.7B
QWEN57 = dict(H=3584, I=2560, E=64, k=8, shared=20480, shared_gate=True)     # Qwen2-57B-A14B
MIXTRAL = dict(H=4096, I=14336, E=8, k=2, norm=True, q4=True)                # Mixtral-8x7B, uint4 group 128


def listed():
    def c(name, kind, T, shape, **more):
        return dict(_case(kind, T, **{**shape, **more}), name=name)
    return [
        # one user typing: a single token through a layer, the latency of every generated token
        c("decode1_v2lite", "layer", 1, DSMOE),
        # the same call through host buffers, four sequences (a serving loop that keeps activations on the host)
        c("decode4_v2lite_host", "host", 4, DSMOE),
        # the benchmark's decode batch of 8, experts resident, next-layer predictors on (two layers)
        c("decode8_qwen_predict", "stack", 8, QWEN, L=2, predict=4),
        # the benchmark's workload in small: cache_rate 0.375, missing experts come over the host link
        c("decode8_qwen_offload", "stack", 8, QWEN, L=2, steps=4, rate=0.375, predict=4),
        # 32 sequences decoded together: experts with a few rows each, a 32-row shared expert
        c("decode32_dsmoe", "layer", 32, DSMOE),
        # large decode batch, top-8: every expert active with 1 to 40 rows, a very wide shared expert
        c("decode64_qwen57", "layer", 64, QWEN57),
        # uint4 experts: one user, and a batch of 16
        c("decode1_mixtral_q4", "layer", 1, MIXTRAL),
        c("decode16_mixtral_q4", "layer", 16, MIXTRAL),
        # owner side of expert parallelism over 4 ranks: 16 tokens in flight, 16 of the 64 experts here
        c("routed16_v2lite_ep4", "routed", 16, DSMOE, world=4),
        # a short chat prompt of odd length: about 50 rows per expert
        c("prompt777_qwen", "layer", 777, QWEN),
        # prompt through uint4 experts
        c("prompt512_mixtral_q4", "layer", 512, MIXTRAL),
        # a batch of long prompts (4 x 2048 tokens)
        c("prompt8192_v2lite", "layer", 8192, DSMOE),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another layer of these ranges: sizes between and around the configurations', any batch."""
    what = rng.choice(["bf16", "bf16", "bf16", "q4", "q4", "routed", "stack"])
    H = 128 * rng.randint(8, 28)
    E = rng.randint(8, 64)
    k = rng.randint(1, min(8, E))
    I = 64 * rng.randint(8, 44)
    if what == "q4":
        H = 256 * rng.randint(4, 16)
        E = rng.randint(4, 16)
        k = rng.randint(1, min(4, E))
        I = 128 * rng.randint(4, 112 if E <= 8 else 40)
        top = 512 if I > 4096 else 2048
        return _case("layer", _log_int(rng, 1, top), H, I, E, k, norm=rng.random() < 0.5, q4=True)
    if what == "routed":
        return _case("routed", _log_int(rng, 1, 256), H, I, E=4 * rng.randint(4, 16), k=min(k, 6), world=4)
    shared = 0 if rng.random() < 0.25 else 64 * rng.randint(8, 96)
    if what == "stack":
        I = 64 * rng.randint(8, 22)
        return _case("stack", _log_int(rng, 1, 32), H, I, E=min(E, 32), k=min(k, 4), shared=shared,
                     shared_gate=rng.random() < 0.5, L=2, steps=rng.randint(1, 4),
                     rate=rng.choice([0.375, 0.5, 1.0, 1.0]), predict=rng.choice([0, 2, 4]))
    # the widest and the longest do not come together
    top = 8192 if H * (k * I + shared) <= 2048 * (6 * 1408 + 2816) else 2048
    return _case(rng.choice(["layer", "layer", "layer", "host"]), _log_int(rng, 1, top), H, I, E, k, shared=shared,
                 shared_gate=shared > 0 and rng.random() < 0.5, norm=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------ inputs
def _gen(seed, *parts):
    h = seed * 1000003 + 17
    for p in parts:
        h = (h * 8191 + p + 1) % (1 << 61)
    return torch.Generator(device="cuda").manual_seed(h)


def _randn(g, *shape, std=STD, dtype=torch.bfloat16):
    return (torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * std).to(dtype)


def _quantise(w):
    """Asymmetric uint4, 128 weights of a row to a group: packed words (the even weights of every eight in the
    low half of the word, the odd ones in the high half) and {scale, zero} fp16 pairs."""
    rows, K = w.shape
    g = w.view(rows, K // 128, 128)
    lo, hi = g.amin(2), g.amax(2)
    scale = ((hi - lo) / 15.0).clamp_min(1e-8).half()
    zero = (-lo / scale.float()).half()
    q = torch.round(g / scale.float()[..., None] + zero.float()[..., None]).clamp_(0, 15).to(torch.int32)
    q = q.view(rows, K // 8, 8)
    word = torch.zeros((rows, K // 8), dtype=torch.int32, device=w.device)
    for j in range(4):
        word |= (q[:, :, 2 * j] << (4 * j)) | (q[:, :, 2 * j + 1] << (4 * j + 16))
    return word, torch.stack([scale, zero], dim=-1).contiguous()


def _dequantise(word, sz):
    rows, n = word.shape
    q = torch.empty((rows, n, 8), dtype=torch.float64, device=word.device)
    for j in range(4):
        q[:, :, 2 * j] = ((word >> (4 * j)) & 15).double()
        q[:, :, 2 * j + 1] = ((word >> (4 * j + 16)) & 15).double()
    q = q.view(rows, n // 16, 128)
    s, z = sz[..., 0].double(), sz[..., 1].double()
    return ((q - z[..., None]) * s[..., None]).view(rows, n * 8)


def _expert_ids(case):
    """The routed experts a context holds: all of them, or one rank's block."""
    return range(case["E"] // case["world"])


def _expert(case, seed, layer, e):
    """Tensors of one expert in the order of the cache's parameter list."""
    H, I = case["H"], case["I"]
    g = _gen(seed, 1, layer, e)
    mats = [_randn(g, *s, dtype=torch.float32 if case["q4"] else torch.bfloat16) for s in ((I, H), (I, H), (H, I))]
    if not case["q4"]:
        return mats
    return [t for m in mats for t in _quantise(m)]


def _layer(case, seed, layer):
    """Router, gate bias (half the log of Zipf(1.1) popularity), shared expert and its sigmoid gate."""
    H, E, Is = case["H"], case["E"], case["shared"]
    g = _gen(seed, 2, layer)
    gate_w = _randn(g, E, H)
    rank = torch.randperm(E, generator=g, device="cuda").double() + 1
    p = rank ** -1.1
    bias = (0.5 * torch.log(p / p.sum())).float()
    shared = [_randn(g, Is, H), _randn(g, Is, H), _randn(g, H, Is)] if Is else None
    return gate_w, bias, shared, _randn(g, H) if case["shared_gate"] and Is else None


def _tokens(case, seed):
    """[steps, T, H] bf16 hidden states: an AR(1) chain per sequence, unit variance."""
    g = _gen(seed, 3)
    h = torch.randn((case["T"], case["H"]), generator=g, device="cuda")
    out = []
    for _ in range(case["steps"]):
        out.append(h.to(torch.bfloat16))
        h = 0.8 * h + 0.6 * torch.randn(h.shape, generator=g, device="cuda")
    return torch.stack(out)


def _routed_rows(case, seed):
    """The receive buffer of one owner: per source rank a header row, then the rows routed to the owner's
    experts in expert order, then unused rows (-1). Returns (x [n, H] bf16, row_expert [n] int32)."""
    world, E, k, H = case["world"], case["E"], case["k"], case["H"]
    per = max(1, -(-case["T"] // world))
    cap = per * k
    gate_w, bias, _, _ = _layer(case, seed, 0)
    x = _tokens(case, seed)[0]
    x = x.repeat(world, 1)[: per * world]
    ids = torch.topk(x.double() @ gate_w.double().T + bias.double(), k, dim=1).indices
    rows = torch.zeros((world * (1 + cap), H), dtype=torch.bfloat16, device="cuda")
    row_expert = torch.full((world * (1 + cap),), -1, dtype=torch.int32, device="cuda")
    for r in range(world):
        mine = ids[r * per:(r + 1) * per]
        tok, slot = torch.nonzero(mine < E // world, as_tuple=True)
        e = mine[tok, slot]
        order = torch.argsort(e, stable=True)
        at = r * (1 + cap) + 1
        rows[at:at + order.numel()] = x[r * per:(r + 1) * per][tok[order]]
        row_expert[at:at + order.numel()] = e[order].to(torch.int32)
    return rows, row_expert


def _pinned(addr, nbytes):
    return torch.frombuffer((ctypes.c_ubyte * nbytes).from_address(addr), dtype=torch.uint8)


def prepare(case, seed):
    H, I, L, q4 = case["H"], case["I"], case["L"], case["q4"]
    experts = list(_expert_ids(case))
    cache = ExpertCache(L, len(experts), num_expert_per_token=case["k"] if case["kind"] != "routed" else 1,
                        cache_rate=repr(case["rate"]), num_predict_expert_per_layer=case["predict"])
    if q4:
        cache.set_param_list(["w1.qweight", "w1.scale_zero", "w3.qweight", "w3.scale_zero", "w2.qweight", "w2.scale_zero"])
        sizes = [I * H // 2, I * H // 128 * 4] * 3
    else:
        cache.set_param_list(["gate_proj.weight", "up_proj.weight", "down_proj.weight"])
        sizes = [I * H * 2] * 3
    for l in range(L):
        for e in experts:
            cache.register_expert_sizes(l, e, sizes)
    cache.pin_all()
    for l in range(L):
        for e in experts:
            for p, t in enumerate(_expert(case, seed, l, e)):
                addr, n = cache.host_record(l, e, p)
                _pinned(addr, n).copy_(t.view(-1).view(torch.uint8))
    cache.build_slab()
    state = dict(case=case, cache=cache, layers=[])
    for l in range(L):
        if case["kind"] == "routed":
            cache.set_layer_weights(l, None, I, 1, False, 1.0, hidden=H)
        else:
            gate_w, bias, shared, sg = _layer(case, seed, l)
            cache.set_layer_weights(l, gate_w, I, case["k"], case["norm"], 1.0, gate_bias=bias, shared=shared,
                                    shared_gate_w=sg, quant4=q4)
        if case["rate"] >= 1.0:  # every expert is resident
            for e in cache.report_layer(l, experts):
                cache.expert_done(l, e)
            cache.layer_done(l)
    if case["predict"]:
        E = case["E"]
        for src in range(L):
            for dst in range(L):
                g = _gen(seed, 4, src, dst)
                cache.set_predictor(src, dst, _randn(g, PRED_D, H), torch.zeros(PRED_D, device="cuda"),
                                    _randn(g, E, PRED_D), torch.zeros(E, device="cuda"))
        cache.set("predict_from_moe_input", 1)
    kind = case["kind"]
    if kind == "routed":
        state["x"], state["row_expert"] = _routed_rows(case, seed)
        state["out"] = torch.empty(state["x"].shape, dtype=torch.float32, device="cuda")
        state["bound"] = max(1, -(-case["T"] // case["world"])) * case["world"]
    elif kind == "host":
        state["x"] = _tokens(case, seed)[0].cpu().pin_memory()
        state["out"] = torch.empty_like(state["x"]).pin_memory()
    else:
        state["x"] = _tokens(case, seed)
    cache.set("seq_len", 1 if kind in ("stack", "routed") or case["T"] <= 64 else case["T"])
    torch.cuda.synchronize()
    return state


def run(state):
    cache, kind, x = state["cache"], state["case"]["kind"], state["x"]
    if kind == "host":
        return cache.forward_host(0, x, out=state["out"])
    if kind == "routed":
        _lib.call("pm_moe_forward_routed", cache.handle, 0, x.data_ptr(), x.shape[0], state["row_expert"].data_ptr(),
                  state["out"].data_ptr(), state["bound"], None, None, 0, 0, 0, 0,
                  torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "layer":
        return cache.forward(0, x[0])
    return [cache.forward(l, x[s]) for s in range(x.shape[0]) for l in range(state["case"]["L"])]


# --------------------------------------------------------------------------------------- arithmetic
def _ffn(x, mats):
    g, u, d = mats
    a = x @ g.T
    return ((a / (1 + torch.exp(-a))) * (x @ u.T)) @ d.T


def exact(case, seed):
    """The layer in 64 bits on the same 16-bit (or uint4) inputs."""
    if case["T"] * case["steps"] * case["L"] * (case["k"] * case["I"] + case["shared"]) * case["H"] > 4e11:
        return None
    f64 = torch.float64

    def matrices(layer, e):
        t = _expert(case, seed, layer, e)
        if case["q4"]:
            return [_dequantise(t[2 * i], t[2 * i + 1]) for i in range(3)]
        return [m.to(f64) for m in t]

    if case["kind"] == "routed":
        rows, row_expert = _routed_rows(case, seed)
        out = torch.zeros(rows.shape, dtype=f64, device="cuda")
        for e in _expert_ids(case):
            at = torch.nonzero(row_expert == e)[:, 0]
            if at.numel():
                out[at] = _ffn(rows[at].to(f64), matrices(0, e))
        return out
    xs = _tokens(case, seed)
    outs = {}
    for l in range(case["L"]):
        gate_w, bias, shared, sg = _layer(case, seed, l)
        x = xs.reshape(-1, case["H"]).to(f64)
        logits = x @ gate_w.to(f64).T + bias.to(f64)
        prob = torch.softmax(logits, dim=1)
        ids = torch.topk(logits, case["k"], dim=1).indices
        w = torch.gather(prob, 1, ids)
        if case["norm"]:
            w = w / w.sum(1, keepdim=True)
        y = torch.zeros_like(x)
        for e in range(case["E"]):
            tok, slot = torch.nonzero(ids == e, as_tuple=True)
            if tok.numel():
                y.index_add_(0, tok, w[tok, slot][:, None] * _ffn(x[tok], matrices(l, e)))
        if shared is not None:
            s = _ffn(x, [m.to(f64) for m in shared])
            y += s * torch.sigmoid(x @ sg.to(f64))[:, None] if sg is not None else s
        outs[l] = y.view(case["steps"], case["T"], case["H"])
    if case["kind"] == "layer":
        return outs[0][0]
    if case["kind"] == "host":
        return outs[0][0].cpu()
    return [outs[l][s] for s in range(case["steps"]) for l in range(case["L"])]


def work(case):
    """Weights of the activated experts read once per layer call, rows in and out once, and the products.
    How many experts a batch activates is counted on random logits of the same distribution."""
    H, I, E, k, T, Is = case["H"], case["I"], case["E"], case["k"], case["T"], case["shared"]
    g = torch.Generator().manual_seed(11)
    p = (torch.arange(E, dtype=torch.float64) + 1) ** -1.1
    logits = torch.randn((T, E), generator=g, dtype=torch.float64) * (STD * math.sqrt(H)) + 0.5 * torch.log(p / p.sum())
    ids = torch.topk(logits, k, dim=1).indices
    unique, pairs = int(torch.unique(ids).numel()), T * k
    if case["kind"] == "routed":
        unique, pairs = max(1, unique // case["world"]), max(1, pairs // case["world"])
    per = 3 * H * I * (0.5 + 4 / 128) if case["q4"] else 6 * H * I
    one = unique * per + 6 * H * Is + T * H * 4
    flops = 6.0 * H * I * pairs + 6.0 * H * Is * T
    if case["kind"] == "routed":
        one = unique * per + pairs * H * 6
    else:
        one += E * H * 2
        flops += 2.0 * T * H * E
    if case["predict"]:
        one += 2 * PRED_D * (H + E)
        flops += 2.0 * T * PRED_D * (H + E)
    n = case["L"] * case["steps"]
    return {"bytes": float(one * n), "flops": float(flops * n)}


def tolerance(case):
    # bf16 intermediate rows and (but for the routed form) bf16 results: about 2e-3 against 64 bits
    return {"rel": 8e-3}
