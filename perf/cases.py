"""The work that a user of this package has it do on one GPU, as cases that can be timed and compared.

A case is a dict of plain values; `kind` names the entry points it goes through:

  ep            Buffer.get_dispatch_layout + dispatch + combine (normal mode), one training or prefill
                exchange; `dtype` is what travels, `mode` whether rows arrive per rank or per expert
  ep_grad       the same exchange through the autograd functions of models.fused_a2a, forward and backward
  ll            Buffer.low_latency_dispatch + low_latency_combine, the decode step; `graph` replays it
                from a CUDA graph as a serving loop does
  experts       Tcgen05GroupedExperts forward (inference), rows already grouped by expert
  experts_fp8   the same with the e4m3 rows and 1x128 scales that an fp8 dispatch delivers
  experts_grad  Tcgen05GroupedExperts forward and backward
  layer         MoELayer forward without gradients: router, dispatch, experts, combine
  layer_grad    MoELayer forward and backward

The sizes are those of the package's benchmarks and tests (7168 x 2048 with 256 experts and top-8,
4096 x 14336 with 8 experts and top-2) and generic ones around them. One GPU is a group of one rank: it
keeps all experts, and every peer address is its own memory.
"""
from __future__ import annotations

import math

import torch

from gpu_data_transfer_profile_b200.models import fused_a2a as A
from gpu_data_transfer_profile_b200.models.experts_tcgen05 import Tcgen05GroupedExperts
from gpu_data_transfer_profile_b200.models.moe_layer import MoELayer
from gpu_data_transfer_profile_b200.ops import gemm as G
from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32, "fp8": torch.bfloat16}
LEAST_ROWS = 512        # rows that an expert has at least in a training batch
NUM_SMS = 132           # CTA budget of the normal-mode kernels, as the headline benchmark sets it


# ------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a small exchange (a few sequences of a small model): launches, the host read of the receive count
        dict(name="ep small", kind="ep", mode="rank", dtype="bf16", tokens=96, hidden=1024, experts=64, topk=8,
             zipf=0.0, worst=False, zero_copy=False, weights=True),
        # the headline exchange of the benchmark: no host read, zero-copy receive rows, pull combine
        dict(name="ep 4096x7168", kind="ep", mode="rank", dtype="bf16", tokens=4096, hidden=7168, experts=256, topk=8,
             zipf=0.0, worst=True, zero_copy=True, weights=False),
        # fp8 on the wire, rows grouped by expert, a skewed router, an odd number of tokens
        dict(name="ep fp8 grouped", kind="ep", mode="expert", dtype="fp8", tokens=2047, hidden=7168, experts=64, topk=8,
             zipf=0.8, worst=False, zero_copy=True, weights=False),
        # the exchange of a training step: dispatch and combine, and each as the other's backward
        dict(name="exchange grad", kind="ep_grad", tokens=4096, hidden=4096, experts=8, topk=2, zipf=0.3),
        # a decode step of a serving loop from a CUDA graph: 128 tokens, the experts of one rank of eight
        dict(name="decode graph fp8", kind="ll", tokens=128, hidden=7168, experts=32, topk=8, fp8=True, graph=True),
        # a few sequences decoding, called eagerly, bf16 rows sent back to their tokens
        dict(name="decode eager", kind="ll", tokens=7, hidden=4096, experts=16, topk=4, fp8=False, graph=False),
        # experts of a decode step: few rows for each expert, all weights are read
        dict(name="experts decode", kind="experts", rows=256, experts=32, hidden=7168, ffn=2048, act="swiglu", skew=0.3),
        # experts of a prefill: thousands of rows for each expert
        dict(name="experts prefill", kind="experts", rows=8191, experts=8, hidden=4096, ffn=14336, act="swiglu", skew=0.3),
        # the fp8 form, rows as an fp8 dispatch delivers them
        dict(name="experts fp8", kind="experts_fp8", rows=8190, experts=32, hidden=7168, ffn=2048, act="swiglu", skew=0.3),
        # forward and backward of many small experts, ragged
        dict(name="experts grad", kind="experts_grad", rows=12001, experts=16, hidden=2048, ffn=1408, act="swiglu", skew=0.5),
        # a whole layer, inference, its own router
        dict(name="layer", kind="layer", tokens=1024, hidden=2048, ffn=1024, experts=64, topk=8, act="swiglu", fp8=False),
        # a whole layer, a training step
        dict(name="layer grad", kind="layer_grad", tokens=4095, hidden=4096, ffn=2048, experts=8, topk=2, act="swiglu"),
    ]


def _log(rng, lo, hi, step=1):
    """A whole number between lo and hi, spread over its logarithm, a multiple of `step`."""
    return max(step, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)


def draw(rng):
    kind = rng.choice(["ep", "ep", "ep_grad", "ll", "ll", "experts", "experts", "experts_fp8", "experts_grad",
                       "layer", "layer_grad"])
    if kind == "ep":
        dtype, mode = rng.choice(["bf16", "bf16", "fp8", "f16", "f32"]), rng.choice(["rank", "expert"])
        topk = rng.choice([1, 2, 4, 6, 8])
        hidden = _log(rng, 256, 7168, 128)
        most = 4096 * 7168 // hidden // (2 if dtype == "f32" else 1) // (topk if mode == "expert" else 1)
        return dict(kind=kind, mode=mode, dtype=dtype, tokens=_log(rng, 8, min(16384, max(64, most))), hidden=hidden,
                    experts=rng.choice([8, 16, 64, 160, 256]), topk=topk, zipf=rng.choice([0.0, 0.5, 1.0]),
                    worst=rng.random() < 0.5, zero_copy=rng.random() < 0.5, weights=rng.random() < 0.5)
    if kind == "ep_grad":
        topk, hidden = rng.choice([1, 2, 4, 8]), _log(rng, 512, 7168, 8)
        return dict(kind=kind, tokens=_log(rng, 16, min(16384, 2 * 4096 * 4096 // (topk * hidden))), hidden=hidden,
                    experts=rng.choice([8, 16, 64, 256]), topk=topk, zipf=rng.choice([0.0, 0.5, 1.0]))
    if kind == "ll":
        return dict(kind=kind, tokens=_log(rng, 1, 160), hidden=_log(rng, 1024, 7168, 128), experts=rng.choice([8, 16, 32, 64]),
                    topk=rng.choice([1, 2, 4, 8]), fp8=rng.random() < 0.5, graph=rng.random() < 0.5)
    if kind in ("layer", "layer_grad"):
        topk, hidden, ffn = rng.choice([1, 2, 4, 8]), _log(rng, 512, 4096, 128), _log(rng, 256, 2048, 128)
        act, experts = rng.choice(["swiglu", "swiglu", "gelu", "silu", "relu"]), rng.choice([8, 16, 32])
        if kind == "layer":
            most = 2048 * 2 * 4096 * 2048 // (topk * hidden * ffn)
            return dict(kind=kind, tokens=_log(rng, 8, min(4096, max(64, most))), hidden=hidden, ffn=ffn,
                        experts=experts, topk=topk, act=act, fp8=rng.random() < 0.3)
        topk = max(2, topk)                          # one choice of weight 1 has no router gradient
        experts = min(experts, 8 * topk)             # a training batch fills its experts
        low = max(768, 768 * experts // topk)
        return dict(kind=kind, tokens=_log(rng, low, max(low, 4095)), hidden=hidden, ffn=ffn, experts=experts, topk=topk, act=act)
    # the expert kinds
    experts, hidden, ffn = rng.choice([1, 4, 8, 16, 32]), _log(rng, 512, 7168, 128), _log(rng, 256, 8192, 128)
    top = {"experts": 8191 * 4096 * 14336, "experts_fp8": 8190 * 7168 * 2048, "experts_grad": 1}[kind]
    low, most = (1 if kind == "experts" else 16), min(16384, max(64, top // (hidden * ffn)))
    if kind == "experts_grad":
        experts, hidden, ffn = rng.choice([1, 4, 8, 16]), _log(rng, 512, 2048, 128), _log(rng, 256, 1408, 128)
        low, most = LEAST_ROWS * experts, 1024 * experts
    return dict(kind=kind, rows=max(low, _log(rng, low, most)),
                experts=experts, hidden=hidden, ffn=ffn, act=rng.choice(["swiglu", "swiglu", "gelu", "silu"]),
                skew=rng.choice([0.0, 0.3, 1.0]))


# ------------------------------------------------------------------------------------------ inputs
def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(1_000_003 * (seed + 1) % (1 << 31))


def _routing(g, T, E, K, zipf):
    """Top-k of a softmax over normal logits plus a Zipf bias over the experts: ids and weights of sum 1."""
    logits = torch.randn(T, E, generator=g, device=g.device)
    if zipf:
        bias = torch.log(torch.arange(1, E + 1, device=g.device, dtype=torch.float32))
        logits = logits - zipf * bias[torch.randperm(E, generator=g, device=g.device)][None]
    w, idx = torch.topk(torch.softmax(logits, -1), K, dim=-1)
    return idx, w / w.sum(-1, keepdim=True)


def _counts(case, seed):
    """Rows of each expert: a multinomial draw, `skew` 0 for an even router. In a training batch the
    balancing loss leaves no expert nearly empty: each has LEAST_ROWS rows and a share of the others."""
    g = _gen(seed, "cpu")
    least = LEAST_ROWS if case["kind"] == "experts_grad" else 0
    p = torch.exp(case["skew"] * torch.randn(case["experts"], generator=g))
    more = case["rows"] - least * case["experts"]
    if more == 0:
        return torch.full((case["experts"],), least)
    pick = torch.multinomial(p, more, replacement=True, generator=g)
    return torch.bincount(pick, minlength=case["experts"]) + least


def _quantise_rows(x):
    xf = x.float().view(x.shape[0], -1, 128)
    amax = xf.abs().amax(-1).clamp_min(1e-4)
    q = (xf * (448.0 / amax)[..., None]).clamp(-448, 448).to(torch.float8_e4m3fn).view(x.shape)
    return q, amax / 448.0


_BUFFER = {}


def _buffer(H, T, K, E, grouped, slots, elem):
    """The program's exchange buffer: made for a shape and used for all inputs of that shape (zero-copy
    outputs are views of it, so it outlives them), given back when another shape comes."""
    key = (H, T, K, E, grouped, slots, elem)
    if key not in _BUFFER:
        for b in _BUFFER.values():
            b.destroy()
        _BUFFER.clear()
        cfg = Buffer.get_dispatch_config(1, T, K, E, group_by_expert=grouped, combine_slots=slots)
        _BUFFER[key] = Buffer(None, cfg.get_nvl_buffer_size_hint(H * elem, 1), 0, world=LocalWorld.make(1)[0],
                              combine_slots=slots)
    return _BUFFER[key]


class _Held:
    """A Buffer that is given back with the state that holds it (no output is a view of it)."""

    def __init__(self, *a, **k):
        self.buf = Buffer(*a, **k)

    def __del__(self):
        self.buf.destroy()


_WORLD = []


def _world():
    """The one-rank group of this process, made once as a program makes its process group."""
    if not _WORLD:
        _WORLD.append(LocalWorld.make(1, torch.device("cuda", torch.cuda.current_device()))[0])
    return _WORLD[0]


def _exchange_inputs(case, seed):
    g = _gen(seed)
    T, H, E, K = (case[k] for k in ("tokens", "hidden", "experts", "topk"))
    x = torch.randn(T, H, generator=g, device="cuda")
    idx, w = _routing(g, T, E, K, case.get("zipf", 0.0))
    return g, T, H, E, K, x, idx, w


def _expert_weights(g, case):
    E, H, F = case["experts"], case["hidden"], case["ffn"]
    n1 = 2 * F if case["act"] == "swiglu" else F
    w1 = torch.randn(E, n1, H, generator=g, device="cuda", dtype=torch.bfloat16) * 0.02
    w2 = torch.randn(E, H, F, generator=g, device="cuda", dtype=torch.bfloat16) * 0.02
    return w1, w2


def _set_weights(m, w1, w2):
    with torch.no_grad():
        m.weight1.copy_(w1)
        m.weight2.copy_(w2)


def _expert_inputs(case, seed):
    g = _gen(seed)
    counts = _counts(case, seed)
    x = torch.randn(case["rows"], case["hidden"], generator=g, device="cuda").to(torch.bfloat16)
    probs = torch.rand(case["rows"], generator=g, device="cuda")
    w1, w2 = _expert_weights(g, case)
    dy = torch.randn(case["rows"], case["hidden"], generator=g, device="cuda").to(torch.bfloat16)
    return counts, x, probs, w1, w2, dy


def _layer_inputs(case, seed):
    g = _gen(seed)
    x = torch.randn(case["tokens"], case["hidden"], generator=g, device="cuda").to(torch.bfloat16)
    router = torch.randn(case["experts"], case["hidden"], generator=g, device="cuda") * 0.02
    logits = torch.randn(case["tokens"], case["experts"], generator=g, device="cuda")
    w1, w2 = _expert_weights(g, case)
    dy = torch.randn(case["tokens"], case["hidden"], generator=g, device="cuda").to(torch.bfloat16)
    return x, router, logits, w1, w2, dy


def prepare(case, seed):
    kind, s = case["kind"], dict(case=case)
    Buffer.set_num_sms(NUM_SMS)
    if kind == "ep":
        g, T, H, E, K, x, idx, w = _exchange_inputs(case, seed)
        dtype, grouped = DTYPES[case["dtype"]], case["mode"] == "expert"
        # the same buffer layout as the headline benchmark: no combine slots where the rows are
        # combined in place
        slots = case["dtype"] == "fp8" or not case["zero_copy"]
        elem = 4 if dtype == torch.float32 else 2
        s.update(buf=_buffer(H, T, K, E, grouped, slots, elem), x=x.to(dtype), idx=idx, w=w)
        if case["dtype"] == "fp8":       # what the experts return: bf16 rows of their own
            n = T * K if grouped else T
            s["y"] = torch.randn(n, H, generator=g, device="cuda").to(torch.bfloat16)
    elif kind == "ep_grad":
        g, T, H, E, K, x, idx, w = _exchange_inputs(case, seed)
        A.configure_buffer(num_max_tokens_per_rank=T, num_topk=K, num_experts=E, group_by_expert=True)
        s.update(x=x.to(torch.bfloat16).requires_grad_(True), idx=idx, w=w.requires_grad_(True),
                 dy=torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16))
    elif kind == "ll":
        g, T, H, E, K, x, idx, w = _exchange_inputs(case, seed)
        held = _Held(None, Buffer.get_low_latency_nvl_size_hint(T, H, 1, E, K), 0, low_latency_mode=True,
                     world=LocalWorld.make(1)[0])
        s.update(held=held, x=x.to(torch.bfloat16), idx=idx, w=w, out=torch.empty(T, H, dtype=torch.bfloat16, device="cuda"))
        if case["fp8"]:
            # the experts write in place; rows arrive in any order, so all rows of an expert are the
            # same here and the sum does not depend on it
            row = torch.randn(E, 1, H, generator=g, device="cuda").to(torch.bfloat16)
            handle = held.buf.low_latency_dispatch(s["x"], idx, T, E, use_fp8=True)[2]
            s["y"] = held.buf.get_next_low_latency_combine_buffer(handle)
            s["y"].copy_(row.expand_as(s["y"]))
            held.buf.low_latency_combine(s["y"], idx, w, handle, out=s["out"])
        if case["graph"]:
            _decode(s)
            torch.cuda.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                s["count"] = _decode(s)[1]
    elif kind in ("experts", "experts_fp8", "experts_grad"):
        counts, x, probs, w1, w2, dy = _expert_inputs(case, seed)
        m = Tcgen05GroupedExperts(case["experts"], case["hidden"], case["ffn"], activation=case["act"],
                                  use_fp8=kind == "experts_fp8")
        _set_weights(m, w1, w2)
        off = G.offsets_from_counts(counts, "cuda")
        s.update(m=m, counts=counts, off=off, x=x, probs=probs)
        if kind == "experts_fp8":
            m.refresh_fp8_weights()
            s["x"] = _quantise_rows(x)
        if kind == "experts_grad":
            s.update(x=x.requires_grad_(True), probs=probs.requires_grad_(True), dy=dy)
    elif kind in ("layer", "layer_grad"):
        x, router, logits, w1, w2, dy = _layer_inputs(case, seed)
        A.configure_buffer(num_max_tokens_per_rank=case["tokens"], num_topk=case["topk"], num_experts=case["experts"],
                           group_by_expert=True)
        m = MoELayer(case["hidden"], case["ffn"], case["experts"], case["topk"], None, activation=case["act"],
                     expert_backend="tcgen05", world=_world(), use_fp8=case.get("fp8", False))
        _set_weights(m.experts, w1, w2)
        with torch.no_grad():
            m.router.weight.copy_(router)
        if case.get("fp8"):
            m.experts.refresh_fp8_weights()
        s.update(m=m, x=x)
        if kind == "layer_grad":
            s.update(x=x.requires_grad_(True), logits=logits.requires_grad_(True), dy=dy)
    else:
        raise ValueError(kind)
    return s


# ------------------------------------------------------------------------------------------ one pass
def _decode(s):
    c, buf = s["case"], s["held"].buf
    recv, count, handle, _, _ = buf.low_latency_dispatch(s["x"], s["idx"], c["tokens"], c["experts"], use_fp8=c["fp8"])
    y = buf.get_next_low_latency_combine_buffer(handle) if c["fp8"] else recv
    out, _, _ = buf.low_latency_combine(y, s["idx"], s["w"], handle, out=s["out"])
    return out, count


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "ep":
        buf, T, K = s["buf"], case["tokens"], case["topk"]
        grouped, fp8 = case["mode"] == "expert", case["dtype"] == "fp8"
        per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(s["idx"], case["experts"])
        recv_x, recv_idx, recv_w, _, handle, _ = buf.dispatch(
            s["x"], topk_idx=s["idx"], topk_weights=s["w"], num_tokens_per_rank=per_rank, is_token_in_rank=in_rank,
            num_tokens_per_expert=per_expert, use_fp8=fp8, group_by_expert=grouped, zero_copy=case["zero_copy"],
            num_worst_tokens=(T * K if grouped else T) if case["worst"] else 0)
        y = s["y"] if fp8 else recv_x
        side = (handle.recv_prob if grouped else recv_w) if case["weights"] else None
        out, out_w, _ = buf.combine(y, handle, topk_weights=side, item_weights=s["w"] if grouped else None)
        return dict(per_rank=per_rank, per_expert=per_expert, in_rank=in_rank, recv_x=recv_x, recv_idx=recv_idx,
                    recv_w=handle.recv_prob if grouped else recv_w, out=out, out_w=out_w)
    if kind == "ep_grad":
        rows, probs, counts, handle = A.FusedDispatchGrouped.apply(s["x"], s["idx"], s["w"], case["experts"], None, _world())
        out = A.FusedCombineGrouped.apply(rows * probs[:, None].to(rows.dtype), None, handle, _world())
        gx, gw = torch.autograd.grad(out, [s["x"], s["w"]], s["dy"])
        return dict(out=out, counts=counts, gx=gx, gw=gw)
    if kind == "ll":
        if case["graph"]:
            s["graph"].replay()
            return dict(out=s["out"], count=s["count"])
        out, count = _decode(s)
        return dict(out=out, count=count)
    if kind == "experts":
        with torch.no_grad():
            return s["m"](s["x"], s["counts"], s["probs"], expert_off=s["off"])
    if kind == "experts_fp8":
        return s["m"].forward_fp8(s["x"], s["counts"], s["probs"], expert_off=s["off"])
    if kind == "experts_grad":
        y = s["m"](s["x"], s["counts"], s["probs"], expert_off=s["off"])
        gx, gp, g1, g2 = torch.autograd.grad(y, [s["x"], s["probs"], s["m"].weight1, s["m"].weight2], s["dy"])
        return dict(y=y, gx=gx, gp=gp, g1=g1, g2=g2)
    if kind == "layer":
        with torch.no_grad():
            return s["m"](s["x"])
    y = s["m"](s["x"], s["logits"])
    ex = s["m"].experts
    gx, gl, g1, g2 = torch.autograd.grad(y, [s["x"], s["logits"], ex.weight1, ex.weight2], s["dy"])
    return dict(y=y, gx=gx, gl=gl, g1=g1, g2=g2)


# ------------------------------------------------------------------------------------------ what a pass costs at least
def work(case):
    kind = case["kind"]
    H = case.get("hidden", 0)
    if kind in ("ep", "ep_grad", "ll"):
        T, K, E = case["tokens"], case["topk"], case["experts"]
        elem = 4 if case.get("dtype") == "f32" else 2
        wire = 1 + 4 / 128 if case.get("dtype") == "fp8" or case.get("fp8") else elem
        n = T if case.get("mode") == "rank" else T * K
        one = T * H * elem + n * H * wire + n * H * elem + T * H * elem + T * K * 24     # out and back
        if kind == "ep_grad":       # forward and backward exchange, and the probabilities in between
            return dict(bytes=2 * one + 6 * n * H * 2, flops=0)
        return dict(bytes=one, flops=0)
    gated = case["act"] == "swiglu"
    F, E = case["ffn"], case["experts"]
    rows = case["rows"] if "rows" in case else case["tokens"] * case["topk"]
    mats = 3 if gated else 2
    touched = E * (1 - (1 - 1 / E) ** rows)               # experts that an even router gives rows
    weights = touched * mats * H * F * 2
    if kind == "experts_fp8" or case.get("fp8"):
        weights = touched * ((mats - 1) * H * F * (1 + 4 / 16384) + H * F * 2)
    flops = 2.0 * rows * mats * H * F
    grad = kind.endswith("grad")
    if "rows" in case:
        acts = rows * H * (2 + (1 + 4 / 128 if kind == "experts_fp8" else 2))
    else:
        acts = 2 * case["tokens"] * H * 2
        flops += 0 if grad else 2.0 * case["tokens"] * H * E
    if grad:
        return dict(bytes=2 * weights + E * mats * H * F * 2 + 2 * acts, flops=3 * flops)
    return dict(bytes=weights + acts, flops=flops)


def tolerance(case):
    kind = case["kind"]
    if kind == "ep":
        # rows are copied; a combine of one row per token is exact too, of several rows it is one
        # rounding to the element type of a sum in f32; fp8 rows are one rounding each
        return {"rel": 1e-6 if case["dtype"] == "f32" else 2e-3, "max": 0.02}
    if kind in ("ep_grad", "ll"):
        return {"rel": 2e-3, "max": 0.05}
    # bf16 products of bf16 roundings in between; a layer's choice of experts may differ at a tie
    return {"rel": 4e-3 if kind.startswith("experts") else 1e-2, "max": 0.2}


# ------------------------------------------------------------------------------------------ in 64 bits
def _act64(h, act):
    F = torch.nn.functional
    if act == "swiglu":
        a, b = h.chunk(2, -1)
        return F.silu(a) * b
    return {"gelu": F.gelu, "silu": F.silu, "relu": F.relu}[act](h)


def _dequantised(w, rows):
    """The values of w (bf16) after e4m3 with one scale per 1 x 128 (rows) or 128 x 128 block."""
    n, k = w.shape[-2:]
    b = w.float().reshape(*w.shape[:-2], n, k // 128, 128) if rows else w.float().reshape(-1, n // 128, 128, k // 128, 128)
    amax = b.abs().amax(-1, keepdim=True) if rows else b.abs().amax((2, 4), keepdim=True)
    amax = amax.clamp_min(1e-4 if rows else 1e-6)
    q = (b * (448.0 / amax)).clamp(-448, 448).to(torch.float8_e4m3fn)
    return (q.double() * (amax / 448.0).double()).reshape(w.shape)


def _mlp64(x, p, w1, w2, act):
    return (_act64(x @ w1.t(), act) * p[:, None]) @ w2.t()


def exact(case, seed):
    kind = case["kind"]
    if kind == "ep":
        g, T, H, E, K, x, idx, w = _exchange_inputs(case, seed)
        grouped, fp8 = case["mode"] == "expert", case["dtype"] == "fp8"
        x = x.to(DTYPES[case["dtype"]]).double()
        w = w.double()
        order = torch.argsort(idx.flatten(), stable=True)
        rows, rw = (x[order // K], w.flatten()[order]) if grouped else (x, w)
        if fp8:
            y = torch.randn(rows.shape[0], H, generator=g, device="cuda").to(torch.bfloat16).double()
            recv = (None, rows.view(rows.shape[0], -1, 128).abs().amax(-1).clamp_min(1e-4) / 448.0)
        else:
            y, recv = rows, rows
        if grouped:
            back = torch.empty_like(y)
            back[order] = y
            out = (back.view(T, K, H) * w[..., None]).sum(1)
        else:
            out = y
        return dict(per_rank=None, per_expert=None, in_rank=None, recv_x=recv, recv_idx=None, recv_w=rw, out=out,
                    out_w=w if case["weights"] else None)
    if kind == "ep_grad":
        g, T, H, E, K, x, idx, w = _exchange_inputs(case, seed)
        x, w = x.to(torch.bfloat16).double(), w.double()
        dy = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16).double()
        total = w.sum(1, keepdim=True)
        return dict(out=x * total, counts=None, gx=dy * total, gw=(dy * x).sum(1, keepdim=True).expand(T, K).contiguous())
    if kind == "ll":
        g, T, H, E, K, x, idx, w = _exchange_inputs(case, seed)
        if case["fp8"]:
            row = torch.randn(E, 1, H, generator=g, device="cuda").to(torch.bfloat16).double()
            out = (row[:, 0][idx] * w.double()[..., None]).sum(1)
        else:
            out = x.to(torch.bfloat16).double() * w.double().sum(1, keepdim=True)
        return dict(out=out, count=None)
    if kind in ("experts", "experts_fp8", "experts_grad"):
        counts, x, p, w1, w2, dy = _expert_inputs(case, seed)
        fp8, grad = kind == "experts_fp8", kind == "experts_grad"
        x = _dequantised(x, True) if fp8 else x.double()
        p = p.double()
        if grad:
            x.requires_grad_(True)
            p.requires_grad_(True)
        ys, g1, g2 = [], [], []
        gx, gp = torch.zeros_like(x), torch.zeros_like(p)
        at = 0
        for e, n in enumerate(counts.tolist()):
            a = (_dequantised(w1[e:e + 1], False)[0] if fp8 else w1[e].double()).requires_grad_(grad)
            b = w2[e].double().requires_grad_(grad)
            xe, pe = x[at:at + n].detach().requires_grad_(grad), p[at:at + n].detach().requires_grad_(grad)
            y = _mlp64(xe, pe, a, b, case["act"])
            ys.append(y.detach())
            if grad:
                d = torch.autograd.grad(y, [xe, pe, a, b], dy[at:at + n].double())
                gx[at:at + n], gp[at:at + n] = d[0], d[1]
                g1.append(d[2])
                g2.append(d[3])
            at += n
        y = torch.cat(ys)
        if not grad:
            return y
        return dict(y=y, gx=gx.detach(), gp=gp.detach(), g1=torch.stack(g1), g2=torch.stack(g2))
    # a whole layer
    x, router, logits, w1, w2, dy = _layer_inputs(case, seed)
    grad, fp8, T, K = kind == "layer_grad", case.get("fp8", False), case["tokens"], case["topk"]
    x64 = x.double()
    logits = logits.double() if grad else x64 @ router.double().t()
    if fp8:
        x64, w1 = _dequantised(x, True), _dequantised(w1, False)
    w1, w2 = w1.double().requires_grad_(grad), w2.double().requires_grad_(grad)
    x64.requires_grad_(grad)
    logits.requires_grad_(grad)
    top, idx = torch.topk(torch.softmax(logits, -1), K, dim=-1)
    probs = top / top.sum(-1, keepdim=True)
    out = torch.zeros_like(x64)
    for e in range(case["experts"]):
        t, k = (idx == e).nonzero(as_tuple=True)
        if t.numel():
            out = out.index_add(0, t, _mlp64(x64[t], probs[t, k], w1[e], w2[e], case["act"]))
    if not grad:
        return out
    d = torch.autograd.grad(out, [x64, logits, w1, w2], dy.double())
    return dict(y=out.detach(), gx=d[0], gl=d[1], g1=d[2], g2=d[3])
