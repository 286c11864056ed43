"""Workloads of this package, timed and compared one call at a time.

A case names one call that a program using the package makes and its sizes; `prepare` builds what
the program holds before the call (weights in their resident layout, inputs, a captured graph),
`run` makes the call. Weights follow the distribution of `bench.py`: N(0, 0.02) with one in a
thousand scaled by 64, so that the coded exponents have outliers as trained weights do.
"""

from __future__ import annotations

import torch

from binade_b200.cuda import kernels, moe, r4

OUTLIERS = 1e-3


def listed() -> list:
    return [
        # One projection of a key or value head group for one token: the smallest product of a
        # decoder layer, called on its own. Its time is the call, not the weights.
        {"name": "linear_1x2048x3840", "op": "linear", "rows": 1, "out": 2048, "in": 3840},
        # One token through all projections of a 12B-class decoder layer, as a decoding loop
        # replays it: projections that share an input in one call, the layer in a CUDA graph.
        {"name": "layer_decode_3840_15360", "op": "layer", "hidden": 3840, "q": 4096, "kv": 2048, "ffn": 15360},
        # Three tokens at once: a short draft being verified, or three sequences in step.
        {"name": "linear_3x15360x3840", "op": "linear", "rows": 3, "out": 15360, "in": 3840},
        # A small serving batch in step, an odd number of sequences, on the layer's long rows.
        {"name": "linear_17x3840x15360", "op": "linear", "rows": 17, "out": 3840, "in": 15360},
        # A chunk of a prompt (or a large batch) on the up projection of an 8B-class layer.
        {"name": "linear_200x14336x4096", "op": "linear", "rows": 200, "out": 14336, "in": 4096},
        # A long prompt.
        {"name": "linear_2048x15360x3840", "op": "linear", "rows": 2048, "out": 15360, "in": 3840},
        # One token through a mixture-of-experts layer, eight experts of 128 (rows of 704: half
        # a tile at their end).
        {"name": "moe_1_token", "op": "moe", "tokens": 1, "experts": 128, "n": 704, "hidden": 2816, "top": 8},
        # A batch of 64 tokens through the same layer: nearly every expert is active.
        {"name": "moe_64_tokens", "op": "moe", "tokens": 64, "experts": 128, "n": 704, "hidden": 2816, "top": 8},
        # Loading a model: one packed matrix from its file arrays to the resident layout.
        {"name": "load_15360x3840", "op": "load", "out": 15360, "in": 3840},
        # Packing a model on the GPU: one BF16 matrix to the file arrays.
        {"name": "pack_15360x3840", "op": "pack", "out": 15360, "in": 3840},
        # Restoring the BF16 weights of an expert stack from the file arrays (rows of 704).
        {"name": "unpack_22528x704", "op": "unpack", "out": 22528, "in": 704},
        # Token rows of a prompt from a table that is kept in its file coding.
        {"name": "embed_300_rice", "op": "embed", "ids": 300, "table": "rice", "out": 32064, "in": 3840},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng) -> dict:
    op = rng.choice(["linear", "linear", "linear", "linear", "layer", "moe", "moe", "load", "pack", "unpack", "embed"])
    wide = lambda lo, hi: 16 * _log(rng, lo // 16, hi // 16)  # noqa: E731 - a row length the fast kernels take
    if op == "linear":
        rows = _log(rng, 1, 2048)
        k = 4 * _log(rng, 160, 3840) if rng.random() < 0.15 else wide(640, 15360)
        n = _log(rng, 704, 16384)
        while n * k > 60_000_000:
            n = n * 3 // 4
        return {"op": op, "rows": rows, "out": n, "in": k}
    if op == "layer":
        hidden = wide(2048, 5120)
        return {"op": op, "hidden": hidden, "q": 128 * rng.randint(16, 40), "kv": 128 * rng.randint(4, 16), "ffn": min(16 * rng.randint(hidden // 8, hidden // 4), 15360)}
    if op == "moe":
        e, n, d = rng.choice([16, 32, 64, 128]), wide(704, 1536), wide(1024, 2816)
        while e * n * d > 128 * 704 * 2816:
            e //= 2
        return {"op": op, "tokens": _log(rng, 1, 64), "experts": e, "n": n, "hidden": d, "top": rng.choice([2, 4, 8])}
    if op == "embed":
        return {"op": op, "ids": _log(rng, 1, 2048), "table": rng.choice(["rice", "r4"]), "out": _log(rng, 4000, 32064), "in": wide(704, 3840)}
    k = wide(704, 15360)
    return {"op": op, "out": max(1, min(_log(rng, 512, 32768), 58_982_400 // k)), "in": k}


def _gen(seed: int, n: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed * 64 + n)


def _weight(shape, g: torch.Generator) -> torch.Tensor:
    w = torch.randn(shape, generator=g, device="cuda").mul_(0.02)
    return torch.where(torch.rand(shape, generator=g, device="cuda") < OUTLIERS, w * 64, w).to(torch.bfloat16)


def _weight_of_one_length(n: int, k: int, g: torch.Generator) -> torch.Tensor:
    """A weight whose coded arrays are as long for every seed: the rows of one fixed matrix in
    another order with other signs."""
    w = _weight((n, k), torch.Generator(device="cuda").manual_seed(n * 31 + k))[torch.randperm(n, generator=g, device="cuda")]
    return torch.where(torch.rand((n, k), generator=g, device="cuda") < 0.5, -w, w)


def _linear(shape, g: torch.Generator) -> r4.R4Linear:
    return r4.R4Linear(r4.from_dense(_weight(shape, g)))


def _x(rows: int, k: int, g: torch.Generator) -> torch.Tensor:
    return torch.randn((rows, k), generator=g, device="cuda").to(torch.bfloat16)


def _layer_shapes(c: dict) -> dict:
    h, f = c["hidden"], c["ffn"]
    return {"q": (c["q"], h), "k": (c["kv"], h), "v": (c["kv"], h), "o": (h, c["q"]), "gate": (f, h), "up": (f, h), "down": (h, f)}


def prepare(case: dict, seed: int) -> dict:
    op, g = case["op"], _gen(seed, 0)
    s = {"op": op}
    if op == "linear":
        s["m"], s["x"] = _linear((case["out"], case["in"]), g), _x(case["rows"], case["in"], g)
    elif op == "layer":
        m = {name: _linear(shape, g) for name, shape in _layer_shapes(case).items()}
        calls = [r4.R4LinearGroup([m[n] for n in names]) for names in (("q", "k", "v"), ("o",), ("gate", "up"), ("down",))]
        xs = [_x(1, k, g) for k in (case["hidden"], case["q"], case["hidden"], case["ffn"])]
        step = lambda: [y for call, x in zip(calls, xs) for y in call(x)]  # noqa: E731
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()
            side.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"], stream=side):
                s["y"] = step()
        torch.cuda.synchronize()
        s["held"] = (m, calls, xs)
    elif op == "moe":
        e, n, d = case["experts"], case["n"], case["hidden"]
        s["m"] = moe.R4SwitchGLU(_linear((e, 2 * n, d), g), _linear((e, d, n), g))
        s["x"] = _x(case["tokens"], d, g)
        s["experts"] = torch.rand((case["tokens"], e), generator=g, device="cuda").topk(case["top"]).indices
    else:
        w = _weight_of_one_length(case["out"], case["in"], g)
        if op == "pack":
            s["w"] = w
            return s
        if op == "embed":
            s["m"] = r4.R4Embedding(r4.from_dense(w)) if case["table"] == "r4" else r4.RiceEmbedding(kernels.rice_encode(w))
            s["ids"] = torch.randint(0, case["out"], (case["ids"],), generator=g, device="cuda")
        else:
            s["w"] = {k: v for k, v in kernels.rice_encode(w).items() if k != "shape"}
    return s


def run(state: dict):
    op = state["op"]
    if op == "linear":
        return state["m"](state["x"])
    if op == "layer":
        state["graph"].replay()
        return state["y"]
    if op == "moe":
        return state["m"](state["x"], state["experts"])
    if op == "load":
        a = r4.transcode(r4.BinadeLinear(state["w"]))
        r4.R4Linear(a)
        return {k: a[k] for k in ("codes", "flags", "esc", "row_esc")}
    if op == "pack":
        p = kernels.rice_encode(state["w"])
        return {k: p[k] for k in ("raw", "table", "meta", "bits", "roff")}
    if op == "unpack":
        w = state["w"]
        n, k = w["raw"].shape
        return kernels.rice_unpack(w["meta"], w["bits"], w["roff"], w["table"], w["raw"], n, k)
    return state["m"](state["ids"])


def _r4_bytes(n: int, k: int) -> float:
    """raw byte, half a code byte of whole tiles, a flag byte a tile, about 0.1 % escapes, an escape cursor a row"""
    t = -(-k // 128)
    return n * (k + 64 * t + t + 0.001 * k + 4)


def _rice_bytes(n: int, k: int) -> float:
    """a tile's meta byte, its stream (2.65 bits a weight on this distribution) and a row offset"""
    return n * (-(-k // 128) + k * 2.65 / 8 + 4)


def work(case: dict) -> dict:
    op = case["op"]
    if op == "linear":
        m, n, k = case["rows"], case["out"], case["in"]
        return {"bytes": _r4_bytes(n, k) + 2 * m * (n + k), "flops": 2.0 * m * n * k}
    if op == "layer":
        shapes = _layer_shapes(case).values()
        return {"bytes": sum(_r4_bytes(n, k) + 2 * n for n, k in shapes) + 2 * (2 * case["hidden"] + case["q"] + case["ffn"]), "flops": sum(2.0 * n * k for n, k in shapes)}
    if op == "moe":
        e, n, d, slots = case["experts"], case["n"], case["hidden"], case["tokens"] * case["top"]
        active = e * (1 - (1 - case["top"] / e) ** case["tokens"])  # experts that some token names
        return {"bytes": active * (_r4_bytes(2 * n, d) + _r4_bytes(d, n)) + 2 * case["tokens"] * d + 2 * slots * d, "flops": 2.0 * slots * 3 * n * d}
    n, k = case["out"], case["in"]
    if op == "load":  # the raw bytes stay where they are
        return {"bytes": _rice_bytes(n, k) + _r4_bytes(n, k) - n * k}
    if op == "embed":
        per_row = _r4_bytes(1, k) if case["table"] == "r4" else k + _rice_bytes(1, k)
        return {"bytes": case["ids"] * (per_row + 2 * k)}
    return {"bytes": 3 * n * k + _rice_bytes(n, k)}  # pack, unpack: BF16 words, raw bytes and the stream


def tolerance(case: dict):
    """Codes, bytes and decoded weights are exact. Products are fp32 sums of exact BF16 products
    rounded once to BF16: against sums in 64 bits, one rounding in 30 at most falls the other way
    by one unit in the last place (relative error 3e-4, largest difference 7.8e-3 over these
    cases); about four times that."""
    if case["op"] in ("load", "pack", "unpack", "embed"):
        return "exact"
    return {"rel": 1.2e-3, "max": 3.1e-2}


def exact(case: dict, seed: int):
    """What `run` gives, in 64 bits from the dense weights; packed arrays have no such value."""
    op, g = case["op"], _gen(seed, 0)
    if op == "linear":
        w, x = _weight((case["out"], case["in"]), g), _x(case["rows"], case["in"], g)
        return x.double() @ w.double().T
    if op == "layer":
        ws = {name: _weight(shape, g) for name, shape in _layer_shapes(case).items()}
        q, o, f, d = (_x(1, k, g).double() for k in (case["hidden"], case["q"], case["hidden"], case["ffn"]))
        return [x @ ws[name].double().T for name, x in (("q", q), ("k", q), ("v", q), ("o", o), ("gate", f), ("up", f), ("down", d))]
    if op == "moe":
        e, n, d, top = case["experts"], case["n"], case["hidden"], case["top"]
        gate_up, down = _weight((e, 2 * n, d), g), _weight((e, d, n), g)
        x = _x(case["tokens"], d, g).double()
        experts = torch.rand((case["tokens"], e), generator=g, device="cuda").topk(top).indices
        y = torch.empty((case["tokens"], top, d), dtype=torch.float64, device="cuda")
        for i in experts.unique().tolist():
            token, slot = torch.nonzero(experts == i, as_tuple=True)
            gate, up = (x[token] @ gate_up[i].double().T).chunk(2, dim=1)
            y[token, slot] = (torch.nn.functional.silu(gate) * up) @ down[i].double().T
        return y
    return None
