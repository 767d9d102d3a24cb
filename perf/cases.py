"""What a program on top of this package has it do, as measurable cases.

Families (the "kind" of a case):

  call     one eager ``lin_forward`` of one linear: a host that drives a layer call by call, where latency counts
  step     a captured decode (or batch-decode / draft-verify) step: the four linears of every layer, replayed as one graph
  multi    the eager decode form for checkpoints that keep q|k|v and gate|up apart (``sk_multi_dev``)
  prefill  the four linears of one layer over a prompt chunk, eager, f16 outputs
  moe      one mixture-of-experts feed-forward layer, from router logits to the summed expert outputs
  head     the int8 lm-head on f32 activations

Weights follow the package's quantiser recipe (N(0, 0.02), absmax / 7 scales); activations are N(0, 1) for decode
and N(0, 1) / sqrt(K) for prefill; router logits are N(0, 1).  Weights are laid out once, in ``prepare``, as a program
that serves a model does; every step streams more weights than the L2 holds.
"""
from __future__ import annotations

import math

import torch

from llm170_b200 import synth
from llm170_b200.w4a16_dec import W4a16Dec

DEV = torch.device("cuda", 0)
F16_OUT = {"rel": 1e-3}      # one rounding to f16 (2^-11 at most, about 3e-4 in the 2-norm) on either side


def _dense(hidden: int, qkv: int, attn: int, ffn: int) -> dict:
    """(K, N) of a layer's four linears."""
    return {"hidden": hidden, "qkv": qkv, "attn": attn, "ffn": ffn}


DENSE_27B = _dense(5120, 7168, 6144, 17408)


def listed():
    return [
        # the smallest call: a one-token linear of an eight-way column shard (qkv of the 27B-class stack), eager
        {"name": "call_shard_t1", "kind": "call", "n": 896, "k": 5120, "group": 128, "bf16": False, "t": 1, "f16": False},
        # a served decode step, one sequence: four layers of the 27B-class stack (0.69 GB of weights)
        {"name": "step_t1", "kind": "step", **DENSE_27B, "layers": 4, "group": 128, "bf16": False, "t": 1},
        # the same for a full small batch, the most rows that the decode path takes
        {"name": "step_t8", "kind": "step", **DENSE_27B, "layers": 4, "group": 128, "bf16": False, "t": 8},
        # batch decode / verification of drafted tokens, just above the decode path's rows; an odd count
        {"name": "step_t27", "kind": "step", **DENSE_27B, "layers": 4, "group": 128, "bf16": False, "t": 27},
        # a small dense model with grouped-query attention and separate projections, bf16 scales in groups of 64
        {"name": "multi_t3_bf16", "kind": "multi", "hidden": 4096, "q": 4096, "kv": 1024, "ffn": 12288, "layers": 4,
         "group": 64, "bf16": True, "t": 3},
        # a short prompt of odd length
        {"name": "prefill_t197", "kind": "prefill", **DENSE_27B, "group": 128, "bf16": False, "t": 197},
        # an ordinary prompt
        {"name": "prefill_t1024", "kind": "prefill", **DENSE_27B, "group": 128, "bf16": False, "t": 1024},
        # a full prefill chunk, the largest case
        {"name": "prefill_t4096", "kind": "prefill", **DENSE_27B, "group": 128, "bf16": False, "t": 4096},
        # one mixture-of-experts layer of the 35B-A3B class: one sequence, a decode batch, a prefill chunk
        {"name": "moe_t1", "kind": "moe", "experts": 128, "local": 128, "top_k": 8, "hidden": 2048, "ffn": 768, "group": 32, "t": 1},
        {"name": "moe_t64", "kind": "moe", "experts": 128, "local": 128, "top_k": 8, "hidden": 2048, "ffn": 768, "group": 32, "t": 64},
        {"name": "moe_t4096", "kind": "moe", "experts": 128, "local": 128, "top_k": 8, "hidden": 2048, "ffn": 768, "group": 32,
         "t": 4096},
        # the logits of one sequence: vocabulary and hidden size of the 35B-A3B-class model
        {"name": "head_t1", "kind": "head", "vocab": 151936, "hidden": 2048, "t": 1},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_dense(rng, tp_most: int) -> dict:
    """Layer shapes of a dense decoder of 3B to 30B parameters, whole or a tensor-parallel shard of it."""
    hidden = 128 * rng.randint(20, 44)
    attn = 128 * max(8, int(hidden * rng.uniform(0.8, 1.25) / 128))
    kv = 128 * rng.choice((4, 8))
    ffn = 128 * int(hidden * rng.uniform(2.4, 3.6) / 128)
    tp = rng.choice([w for w in (1, 1, 1, 2, 4, 8) if w <= tp_most])
    cut = lambda v, unit: max(unit, v // tp // unit * unit)  # noqa: E731
    return _dense(hidden, cut(attn + 2 * kv, 16), cut(attn, 128), cut(ffn, 128))


def _scales(rng) -> dict:
    return {"group": rng.choice((128, 128, 128, 64, 32)), "bf16": rng.random() < 0.25}


def draw(rng):
    kind = rng.choice(("call", "step", "step", "step", "multi", "prefill", "prefill", "prefill", "moe", "moe", "moe", "head"))
    if kind == "call":
        return {"kind": kind, "n": 16 * _log(rng, 32, 512), "k": 128 * rng.randint(12, 48), **_scales(rng),
                "t": _log(rng, 1, 64), "f16": rng.random() < 0.5}
    if kind == "step":
        d = _draw_dense(rng, 8)
        # enough layers that a step streams well over the L2 (126 MB), at most what the listed steps stream
        layers = max(1, min(12, -(-400_000_000 // _layer_bytes(d, 128, 1))))
        return {"kind": kind, **d, "layers": layers, **_scales(rng), "t": rng.choice((1, 1, rng.randint(2, 8), _log(rng, 9, 64)))}
    if kind == "multi":
        hidden = 128 * rng.randint(16, 40)
        return {"kind": kind, "hidden": hidden, "q": hidden, "kv": 128 * rng.choice((2, 4, 8)), "ffn": 128 * int(hidden * rng.uniform(2.4, 3.6) / 128),
                "layers": 3, **_scales(rng), "t": rng.randint(1, 8)}
    if kind == "prefill":
        return {"kind": kind, **_draw_dense(rng, 4), **_scales(rng), "t": _log(rng, 65, 3000)}
    if kind == "moe":
        experts = rng.choice((64, 128, 128, 256))
        return {"kind": kind, "experts": experts, "local": experts // rng.choice((1, 1, 2, 4)), "top_k": rng.choice((4, 6, 8, 8)),
                "hidden": 256 * rng.randint(4, 12), "ffn": 64 * rng.randint(6, 16), "group": rng.choice((32, 32, 64)), "t": _log(rng, 1, 3000)}
    return {"kind": kind, "vocab": 16 * rng.randint(2000, 9496), "hidden": 128 * rng.randint(12, 32), "t": rng.choice((1, 1, rng.randint(2, 16)))}


def _shapes(case) -> list:
    """(name, N, K) of the linears of one layer, in the order they are called."""
    h = case["hidden"]
    if case["kind"] == "multi":
        return [("q", case["q"], h), ("k", case["kv"], h), ("v", case["kv"], h), ("o_proj", h, case["q"]),
                ("gate", case["ffn"], h), ("up", case["ffn"], h), ("down", h, case["ffn"])]
    return [("qkv", case["qkv"], h), ("o_proj", h, case["attn"]), ("gate_up", 2 * case["ffn"], h), ("down", h, case["ffn"])]


def _layer_bytes(dims: dict, group: int, t: int) -> int:
    return sum(synth.decode_bytes(n, k, t, group) for _, n, k in _shapes({"kind": "step", **dims}))


def _randn(shape, seed: int, scale: float = 1.0) -> torch.Tensor:
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return torch.randn(shape, generator=gen, device=DEV, dtype=torch.float32) * scale


def _upload(dec: W4a16Dec, name: str, n: int, k: int, case, seed: int):
    q, s = synth.make_linear_cuda(n, k, case["group"], seed, DEV)
    if case["bf16"]:
        s = s.to(torch.bfloat16)
    dec.upload_lin_g_dev(name, q, s, n, k, case["group"], case["bf16"])


class _Step:
    """A captured step: owns its linears in the process's decoder, its buffers and its graph."""

    dec = None      # one decoder, and so one stream, for all of them, as in a program that serves one device
    made = 0

    def __init__(self, case, seed: int):
        if _Step.dec is None:
            _Step.dec = W4a16Dec(0)
        dec, t = _Step.dec, case["t"]
        _Step.made += 1
        self.names, self.calls, self.graph = [], [], None
        for li in range(case["layers"]):
            for i, (nm, n, k) in enumerate(_shapes(case)):
                name = f"step{_Step.made}.l{li}.{nm}"
                _upload(dec, name, n, k, case, seed * 1000 + li * 8 + i)
                self.names.append(name)
                x = _randn((t, k), seed * 1000 + 500 + li * 8 + i).to(torch.float16)
                self.calls.append((name, x, torch.empty((t, n), device=DEV, dtype=torch.float16)))
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.ExternalStream(dec.stream_ptr(), device=DEV)):
            self._layers(dec, t)            # sizes the decoder's scratch: a capture may not allocate
            dec.sync()
            dec.capture_begin()
            self._layers(dec, t)
            self.graph = dec.capture_end()

    def _layers(self, dec: W4a16Dec, t: int):
        for name, x, y in self.calls:
            dec.lin_forward(name, x, t, dst=y, out_f16=True)

    def run(self):
        self.dec.graph_launch(self.graph)
        return [y for _, _, y in self.calls]

    def __del__(self):
        try:
            self.dec.sync()
            if self.graph is not None:
                self.dec.graph_destroy(self.graph)
            for name in self.names:
                self.dec.drop_lin(name)
        except Exception:
            pass


def prepare(case, seed: int):
    kind = case["kind"]
    if kind == "step":
        return {"kind": kind, "step": _Step(case, seed)}
    dec, t = W4a16Dec(0), case["t"]
    state = {"kind": kind, "dec": dec, "t": t}
    if kind == "call":
        _upload(dec, "lin", case["n"], case["k"], case, seed * 1000)
        state.update(x=_randn((t, case["k"]), seed * 1000 + 1).to(torch.float16), f16=case["f16"])
    elif kind == "prefill":
        state["calls"] = []
        for i, (nm, n, k) in enumerate(_shapes(case)):
            _upload(dec, nm, n, k, case, seed * 1000 + i)
            x = _randn((t, k), seed * 1000 + 500 + i, k ** -0.5).to(torch.float16)
            state["calls"].append((nm, x, torch.empty((t, n), device=DEV, dtype=torch.float16)))
    elif kind == "multi":
        state["layers"] = []
        for li in range(case["layers"]):
            y = {}
            for i, (nm, n, k) in enumerate(_shapes(case)):
                _upload(dec, f"l{li}.{nm}", n, k, case, seed * 1000 + li * 8 + i)
                y[nm] = torch.empty((t, n), device=DEV, dtype=torch.float16)
            x = [_randn((t, k), seed * 1000 + 500 + li * 4 + j).to(torch.float16)
                 for j, k in enumerate((case["hidden"], case["q"], case["hidden"], case["ffn"]))]
            state["layers"].append((x, y))
    elif kind == "moe":
        ne, f, h, g = case["local"], case["ffn"], case["hidden"], case["group"]
        dec.set_moe(case["experts"], case["top_k"], f, h, g, 0, ne)
        q13, s13 = synth.make_linear_cuda(ne * 2 * f, h, g, seed * 1000, DEV)
        q2, s2 = synth.make_linear_cuda(ne * h, f, g, seed * 1000 + 1, DEV)
        dec.upload_experts(0, q13, s13, q2, s2)
        state.update(logits=_randn((t, case["experts"]), seed * 1000 + 2), x=_randn((t, h), seed * 1000 + 3).to(torch.float16))
    else:
        w = _randn((case["vocab"], case["hidden"]), seed * 1000, 0.02).to(torch.bfloat16)
        dec.upload_head(w.view(torch.int16).cpu().numpy().view("uint16"), case["vocab"], case["hidden"])
        state["x"] = _randn((t, case["hidden"]), seed * 1000 + 1)
    return state


def run(state):
    kind = state["kind"]
    if kind == "step":
        return state["step"].run()
    dec, t = state["dec"], state["t"]
    if kind == "call":
        return dec.lin_forward("lin", state["x"], t, out_f16=state["f16"])
    if kind == "prefill":
        return [dec.lin_forward(nm, x, t, dst=y, out_f16=True) for nm, x, y in state["calls"]]
    if kind == "multi":
        outs = []
        for li, (x, y) in enumerate(state["layers"]):
            p = f"l{li}."
            outs += dec.sk_multi_dev([p + "q", p + "k", p + "v"], x[0], [y["q"], y["k"], y["v"]], t=t, out_f16=True)
            outs.append(dec.sk_single_dev(p + "o_proj", x[1], out=y["o_proj"], t=t, out_f16=True))
            outs += dec.sk_multi_dev([p + "gate", p + "up"], x[2], [y["gate"], y["up"]], t=t, out_f16=True)
            outs.append(dec.sk_single_dev(p + "down", x[3], out=y["down"], t=t, out_f16=True))
        return outs
    if kind == "moe":
        return dec.moe_ffn_dev_t(0, state["logits"], state["x"], t)
    return dec.head_forward(state["x"], t)


def work(case):
    kind, t = case["kind"], case["t"]
    if kind == "call":
        n, k = case["n"], case["k"]
        return {"bytes": synth.decode_bytes(n, k, t, case["group"]) + (0 if case["f16"] else 2 * t * n), "flops": synth.gemm_flops(n, k, t)}
    if kind == "head":
        n, k = case["vocab"], case["hidden"]
        return {"bytes": n * k + 4 * n + 4 * t * (k + n), "flops": 2 * n * k * t}
    if kind == "moe":
        ne, local, f, h, g = case["experts"], case["local"], case["ffn"], case["hidden"], case["group"]
        rows = t * case["top_k"] * local / ne                            # rows of the local experts, on average
        hit = local * (1 - (1 - case["top_k"] / ne) ** t)               # local experts with at least one token, on average
        weights = hit * (3 * f * h // 2 + 2 * (2 * f * (h // g) + h * (f // g)))
        return {"bytes": weights + t * (4 * ne + 2 * h + 4 * h), "flops": 2 * rows * 3 * f * h}
    layers = case.get("layers", 1)
    shapes = _shapes(case)
    return {"bytes": layers * sum(synth.decode_bytes(n, k, t, case["group"]) for _, n, k in shapes),
            "flops": layers * sum(synth.gemm_flops(n, k, t) for _, n, k in shapes)}


def tolerance(case):
    kind = case["kind"]
    if kind == "head":
        return {"rel": 1e-5}                  # f32 sums of exact integers times activations carried to 2^-22
    if kind == "moe":
        return {"rel": 2e-3}                  # f16 activations between the two matmuls, f16 expert outputs
    if kind == "call" and not case["f16"]:
        return {"rel": 1e-5} if case["t"] <= 8 else F16_OUT   # above 8 rows the weights are rounded to f16
    return F16_OUT
