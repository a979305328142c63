"""What a user of this library has it do, as cases that can be timed and compared: products with
block-quantized weights, one call or one model step per pass, through the public entry points.

Kinds of cases (each stands for one real use):
  matvec    one decode-time matrix-vector product (qm_matvec), 1..8 activation rows
  ffn       the gated feed-forward block of a decode step, matrix by matrix: gate and up on the RMS-normalised
            input, down on silu(gate) * up (three qm_matvec calls)
  step      a decode step over a stack of layers as one call with pinned host buffers (qm_stack_step_host)
  matmul    a prefill / batched product with bf16 activations (qm_matmul_bf16)
  moe       a mixture-of-experts layer over a batch of tokens: router, then the grouped expert matmuls
  moe_step  the same layer at decode time: router, then the experts of one to a few tokens
  selected  a decode step of a layer whose routed experts are in the low-bit formats, in the Q8_1 activation form:
            RMSNorm to Q8_1, gate and up of the selected experts, SwiGLU to Q8_1, down of the selected experts

Weights are random tensors with the value distributions of lib_b200.synth, made on the GPU. A pass works on weights,
inputs and buffers that it finds in its state; states of different seeds share nothing but the library context.
"""
import functools

import torch

import lib_b200
from lib_b200 import _capi

Q4_0, Q8_0, Q2_K, Q4_K, IQ2_XXS = _capi.Q4_0, _capi.Q8_0, _capi.Q2_K, _capi.Q4_K, _capi.IQ2_XXS
FORMATS = {"q4_0": Q4_0, "q8_0": Q8_0, "q2_k": Q2_K, "q4_k": Q4_K, "iq2_xxs": IQ2_XXS}
# elements and bytes of a block, where its fp16 factors lie and how many they are, and their magnitude
BLOCKS = {Q4_0: (32, 18, 0, 1, 0.004), Q8_0: (32, 34, 0, 1, 0.002), Q4_K: (256, 144, 0, 2, 0.003),
          Q2_K: (256, 84, 80, 2, 0.01), IQ2_XXS: (256, 66, 0, 1, 0.01)}


def listed():
    return [
        # the smallest call: one square matrix of a 4096-wide model, one token
        {"name": "q8_0 matvec", "kind": "matvec", "format": "q8_0", "rows": 4096, "cols": 4096, "m": 1, "xop": 0},
        # an odd one: rows that are no whole tiles, a K of nine super-blocks, three tokens, RMSNorm fused
        {"name": "q4_k matvec ragged", "kind": "matvec", "format": "q4_k", "rows": 10007, "cols": 2304, "m": 3, "xop": 1},
        # the feed-forward block of an 8B-parameter model in Q4_0, single stream and a batch of eight
        {"name": "q4_0 ffn m1", "kind": "ffn", "format": "q4_0", "hidden": 4096, "ffn": 14336, "m": 1},
        {"name": "q4_0 ffn m8", "kind": "ffn", "format": "q4_0", "hidden": 4096, "ffn": 14336, "m": 8},
        # the whole decode step of an 8B-parameter model in Q4_K, single stream and a batch of eight
        {"name": "step m1", "kind": "step", "layers": 32, "hidden": 4096, "kv": 1024, "ffn": 14336, "m": 1},
        {"name": "step m8", "kind": "step", "layers": 32, "hidden": 4096, "kv": 1024, "ffn": 14336, "m": 8},
        # prefill products: a short prompt, an odd length, a long prompt
        {"name": "matmul 64", "kind": "matmul", "rows": 4096, "cols": 4096, "m": 64},
        {"name": "matmul 391", "kind": "matmul", "rows": 6144, "cols": 4096, "m": 391},
        {"name": "matmul 2048", "kind": "matmul", "rows": 4096, "cols": 4096, "m": 2048},
        # a layer of eight experts, top 2: a batch of 512 tokens, and two tokens at decode time
        {"name": "moe 512", "kind": "moe", "experts": 8, "topk": 2, "hidden": 4096, "ffn": 14336, "tokens": 512},
        {"name": "moe step 2", "kind": "moe_step", "experts": 8, "topk": 2, "hidden": 4096, "ffn": 14336, "tokens": 2},
        # six of 64 small experts, IQ2_XXS gate and up, Q2_K down, Q8_1 activations
        {"name": "selected 6 of 64", "kind": "selected", "experts": 64, "slots": 6, "hidden": 4096, "ffn": 2048},
    ]


def draw(rng):
    def log(lo, hi, step=1):
        """A multiple of `step` between lo and hi, even over the logarithm."""
        v = lo * (hi / lo) ** rng.random()
        return max(lo, min(hi, int(round(v / step)) * step))

    kind = rng.choice(["matvec", "matvec", "ffn", "step", "step", "matmul", "matmul", "moe", "moe_step", "selected"])
    if kind == "matvec":
        fmt = rng.choice(["q8_0", "q4_0", "q4_k"])
        return {"kind": kind, "format": fmt, "rows": log(1024, 32768), "cols": log(1024, 14336, 256 if fmt == "q4_k" else 32),
                "m": rng.randint(1, 8), "xop": rng.randint(0, 1)}
    if kind == "ffn":
        return {"kind": kind, "format": rng.choice(["q8_0", "q4_0", "q4_k"]), "hidden": log(1024, 8192, 256),
                "ffn": log(2048, 14336, 256), "m": rng.randint(1, 8)}
    if kind == "step":
        hidden = log(1024, 4096, 256)
        return {"kind": kind, "layers": log(4, 32), "hidden": hidden, "kv": hidden // rng.choice([1, 4, 8]),
                "ffn": log(2048, 14336, 256), "m": rng.randint(1, 8)}
    if kind == "matmul":
        return {"kind": kind, "rows": log(1024, 14336), "cols": log(1024, 14336, 256), "m": log(9, 2048)}
    if kind == "moe":
        return {"kind": kind, "experts": rng.choice([4, 8, 16, 64]), "topk": rng.randint(1, 4), "hidden": log(1024, 4096, 256),
                "ffn": log(1024, 14336, 256) if rng.random() < 0.5 else log(1024, 4096, 256), "tokens": log(32, 1024)}
    if kind == "moe_step":
        return {"kind": kind, "experts": rng.choice([4, 8, 16]), "topk": rng.randint(1, 4), "hidden": log(1024, 4096, 256),
                "ffn": log(1024, 14336, 256), "tokens": rng.randint(1, 8)}
    return {"kind": kind, "experts": rng.choice([16, 64]), "slots": rng.randint(1, 8), "hidden": log(1024, 4096, 256),
            "ffn": log(512, 4096, 256)}


def stored_bytes(fmt, rows, cols):
    elements, size = BLOCKS[fmt][:2]
    return rows * (cols // elements) * size


@functools.lru_cache(maxsize=None)
def context():
    """The program's one library context."""
    torch.cuda.init()
    return lib_b200.Context(0)


class Owned:
    """The library objects of one state, given back with it."""

    def __init__(self):
        self.last = []

    def keep(self, obj, close):
        self.last.append(lambda: close(obj))
        return obj

    def __del__(self):
        for close in reversed(self.last):
            close()


class Maker:
    """Makes tensors and stored matrices from one seed."""

    def __init__(self, seed):
        self.ctx = context()
        self.owned = Owned()
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda")

    def tensor_bytes(self, fmt, rows, cols):
        """The bytes of a rows x cols tensor as a GGUF file holds them."""
        elements, size, at, factors, scale = BLOCKS[fmt]
        blocks = rows * (cols // elements)
        words = torch.randint(-2 ** 63, 2 ** 63 - 1, ((blocks * size + 7) // 8,), generator=self.g, device="cuda")
        raw = words.view(torch.uint8)[:blocks * size].view(blocks, size)
        if fmt == Q8_0:
            raw[:, 2:][raw[:, 2:] == 0x80] = 0   # codes lie in [-127, 127]
        raw[:, at:at + 2 * factors] = (self.normal(blocks, factors).abs() * scale).to(torch.float16).view(torch.uint8)
        return raw.view(-1)

    def weight(self, fmt, rows, cols):
        raw = self.tensor_bytes(fmt, rows, cols)
        w = self.owned.keep(self.ctx.store_create(fmt, rows, cols), lambda w: w.free())
        torch.cuda.synchronize()
        w.write_rows_device(0, rows, raw.data_ptr(), raw.numel())
        self.ctx.sync()
        return w


def prepare(case, seed):
    return PREPARE[case["kind"]](case, Maker(seed))


def run(state):
    return state["pass"](state)


def prepare_matvec(case, make):
    rows, cols, m = case["rows"], case["cols"], case["m"]
    return {"pass": run_matvec, "owned": make.owned, "ctx": make.ctx, "w": make.weight(FORMATS[case["format"]], rows, cols),
            "m": m, "xop": case["xop"], "x": make.normal(m, cols), "y": torch.empty(m, rows, device="cuda")}


def run_matvec(s):
    x, y = s["x"], s["y"]
    s["ctx"].matvec(s["w"], x.data_ptr(), s["m"], x.shape[1], y.data_ptr(), y.shape[1], s["xop"])
    return y


def prepare_ffn(case, make):
    fmt, hidden, ffn, m = FORMATS[case["format"]], case["hidden"], case["ffn"], case["m"]
    return {"pass": run_ffn, "owned": make.owned, "ctx": make.ctx, "m": m, "hidden": hidden, "ffn": ffn,
            "gate": make.weight(fmt, ffn, hidden), "up": make.weight(fmt, ffn, hidden), "down": make.weight(fmt, hidden, ffn),
            "x": make.normal(m, hidden), "g": torch.empty(m, ffn, device="cuda"), "u": torch.empty(m, ffn, device="cuda"),
            "y": torch.empty(m, hidden, device="cuda")}


def run_ffn(s):
    ctx, m, hidden, ffn = s["ctx"], s["m"], s["hidden"], s["ffn"]
    x, g, u = s["x"].data_ptr(), s["g"].data_ptr(), s["u"].data_ptr()
    ctx.matvec(s["gate"], x, m, hidden, g, ffn, _capi.XOP_RMSNORM)
    ctx.matvec(s["up"], x, m, hidden, u, ffn, _capi.XOP_RMSNORM)
    ctx.matvec(s["down"], g, m, ffn, s["y"].data_ptr(), hidden, _capi.XOP_SWIGLU, x2_dev=u)
    return {"gate": s["g"], "up": s["u"], "y": s["y"]}


def prepare_step(case, make):
    layers, hidden, kv, ffn, m = (case[k] for k in ("layers", "hidden", "kv", "ffn", "m"))
    shapes = [(hidden + 2 * kv, hidden), (hidden, hidden), (2 * ffn, hidden), (hidden, ffn)]
    weights = [[make.weight(Q4_K, r, c) for r, c in shapes] for _ in range(layers)]
    stack = make.owned.keep(_capi.Stack(make.ctx, layers, hidden, kv, ffn, m), lambda s: s.close())
    for layer, four in enumerate(weights):
        stack.set_layer(layer, *four)
    pinned = [torch.empty(*shape, pin_memory=True) for shape in ((m, hidden), (m, hidden), (layers, m, 2 * kv))]
    pinned[0].copy_(make.normal(m, hidden))
    x, h, k_v = (t.numpy() for t in pinned)
    return {"pass": run_step, "owned": make.owned, "pinned": pinned, "stack": stack, "x": x, "h": h, "kv": k_v}


def run_step(s):
    return s["stack"].step_host(s["x"], True, s["h"], s["kv"])


def prepare_matmul(case, make):
    rows, cols, m = case["rows"], case["cols"], case["m"]
    return {"pass": run_matmul, "owned": make.owned, "ctx": make.ctx, "w": make.weight(Q4_K, rows, cols),
            "a": make.normal(m, cols).to(torch.bfloat16), "c": torch.empty(m, rows, device="cuda")}


def run_matmul(s):
    a, c = s["a"], s["c"]
    s["ctx"].matmul_bf16(s["w"], a.data_ptr(), a.shape[0], a.shape[1], c.data_ptr(), c.shape[1])
    return c


def experts_of(case, make):
    hidden, ffn, n = case["hidden"], case["ffn"], case["experts"]
    return ([make.weight(Q4_K, 2 * ffn, hidden) for _ in range(n)], [make.weight(Q4_K, hidden, ffn) for _ in range(n)])


def routed(case, make):
    """Router logits of the tokens, and room for the router's answer and the layer's."""
    tokens, topk = case["tokens"], case["topk"]
    return {"owned": make.owned, "ctx": make.ctx, "tokens": tokens, "topk": topk, "hidden": case["hidden"],
            "logits": make.normal(tokens, case["experts"]), "ids": torch.empty(tokens, topk, dtype=torch.int32, device="cuda"),
            "weights": torch.empty(tokens, topk, device="cuda"), "out": torch.empty(tokens, case["hidden"], device="cuda")}


def route(s):
    n = s["logits"].shape[1]
    s["ctx"].moe_route(s["logits"].data_ptr(), s["tokens"], n, n, s["topk"], s["ids"].data_ptr(), s["weights"].data_ptr())


def prepare_moe(case, make):
    gate_up, down = experts_of(case, make)
    return dict(routed(case, make), **{"pass": run_moe, "gate_up": gate_up, "down": down,
                                       "x": make.normal(case["tokens"], case["hidden"]).to(torch.bfloat16)})


def run_moe(s):
    route(s)
    s["ctx"].moe_grouped(s["gate_up"], s["down"], s["x"].data_ptr(), s["tokens"], s["hidden"], s["ids"].data_ptr(),
                         s["weights"].data_ptr(), s["topk"], s["out"].data_ptr(), s["hidden"])
    return {"ids": s["ids"], "weights": s["weights"], "out": s["out"]}


def prepare_moe_step(case, make):
    gate_up, down = experts_of(case, make)
    md = make.owned.keep(make.ctx.moe_decode_create(gate_up, down, case["topk"], case["tokens"]), make.ctx.moe_decode_destroy)
    return dict(routed(case, make), **{"pass": run_moe_step, "gate_up": gate_up, "down": down, "md": md,
                                       "x": make.normal(case["tokens"], case["hidden"])})


def run_moe_step(s):
    route(s)
    s["ctx"].moe_decode_run(s["md"], s["x"].data_ptr(), s["tokens"], s["hidden"], s["ids"].data_ptr(), s["weights"].data_ptr(),
                            s["out"].data_ptr(), s["hidden"])
    return {"ids": s["ids"], "weights": s["weights"], "out": s["out"]}


def prepare_selected(case, make):
    n, slots, hidden, ffn = case["experts"], case["slots"], case["hidden"], case["ffn"]
    order = torch.randperm(n, generator=make.g, device="cuda")[:slots].to(torch.int32)
    blocks = lambda count: torch.zeros(count * 36, dtype=torch.uint8, device="cuda")
    share = torch.rand(slots, generator=make.g, device="cuda") + 0.1
    return {"pass": run_selected, "owned": make.owned, "ctx": make.ctx, "experts": n, "slots": slots, "hidden": hidden, "ffn": ffn,
            "gate": make.weight(IQ2_XXS, n * ffn, hidden), "up": make.weight(IQ2_XXS, n * ffn, hidden),
            "down": make.weight(Q2_K, n * hidden, ffn), "ids": order, "share": share / share.sum(),
            "x": make.normal(1, hidden), "norm": torch.rand(hidden, generator=make.g, device="cuda") + 0.5,
            "xq": blocks(hidden // 32), "hq": blocks(slots * ffn // 32), "g": torch.empty(slots, ffn, device="cuda"),
            "u": torch.empty(slots, ffn, device="cuda"), "y": torch.empty(slots, hidden, device="cuda")}


def run_selected(s):
    ctx, n, slots, hidden, ffn = s["ctx"], s["experts"], s["slots"], s["hidden"], s["ffn"]
    ids, xq, hq, g, u = (s[k].data_ptr() for k in ("ids", "xq", "hq", "g", "u"))
    ctx.rmsnorm_q8_1(s["x"].data_ptr(), hidden, s["norm"].data_ptr(), 1, hidden, 1e-6, xq)
    ctx.matvec_selected(s["gate"], n, ids, slots, xq, 0, g, _capi.FLAG_X_Q8_1)
    ctx.matvec_selected(s["up"], n, ids, slots, xq, 0, u, _capi.FLAG_X_Q8_1)
    ctx.swiglu_q8_1(g, u, s["share"].data_ptr(), ffn, slots, hq)
    ctx.matvec_selected(s["down"], n, ids, slots, hq, ffn // 32, s["y"].data_ptr(), _capi.FLAG_X_Q8_1)
    return {"gate": s["g"], "up": s["u"], "y": s["y"]}


PREPARE = {"matvec": prepare_matvec, "ffn": prepare_ffn, "step": prepare_step, "matmul": prepare_matmul, "moe": prepare_moe,
           "moe_step": prepare_moe_step, "selected": prepare_selected}


def touched(experts, picks):
    """Experts that `picks` independent choices are expected to reach."""
    return experts * (1 - (1 - 1 / experts) ** picks)


def work(case):
    """Each weight byte, input and output once; two operations per weight and token."""
    kind, m = case["kind"], case.get("m", case.get("tokens", case.get("slots")))
    if kind in ("matvec", "matmul"):
        n, k = case["rows"], case["cols"]
        fmt = FORMATS[case["format"]] if kind == "matvec" else Q4_K
        return {"bytes": stored_bytes(fmt, n, k) + m * k * (4 if kind == "matvec" else 2) + m * n * 4, "flops": 2 * m * n * k}
    hidden, ffn = case["hidden"], case["ffn"]
    if kind == "ffn":
        return {"bytes": 3 * stored_bytes(FORMATS[case["format"]], ffn, hidden) + m * (2 * hidden + 2 * ffn) * 4,
                "flops": 6 * m * hidden * ffn}
    if kind == "step":
        elements = case["layers"] * (hidden * (2 * hidden + 2 * case["kv"]) + 3 * hidden * ffn)
        return {"bytes": stored_bytes(Q4_K, 1, elements) + m * (2 * hidden + case["layers"] * 2 * case["kv"]) * 4,
                "flops": 2 * m * elements}
    if kind == "selected":
        return {"bytes": m * (2 * stored_bytes(IQ2_XXS, ffn, hidden) + stored_bytes(Q2_K, hidden, ffn)) + m * (2 * ffn + hidden) * 4 + hidden * 8,
                "flops": 6 * m * hidden * ffn}
    picks = m * case["topk"]
    return {"bytes": touched(case["experts"], picks) * stored_bytes(Q4_K, 3 * ffn, hidden) + m * hidden * (6 if kind == "moe" else 8),
            "flops": 6 * picks * hidden * ffn}


def tolerance(case):
    """About four times the distance from the same pass in float64 on the dequantized weights (listed and drawn cases;
    `selected`: what a float32 sum in another order can change through the rounding of the next Q8_1 blocks)."""
    kind = case["kind"]
    if kind in ("matvec", "ffn"):
        # activations enter with 21 bits of their group's maximum for one and two rows (seen: 7e-7 after one product,
        # 1.7e-6 after two), with 14 bits beyond (1.1e-4, 4e-4)
        few = case["m"] <= 2
        return {"rel": (3e-6 if few else 4e-4) if kind == "matvec" else (8e-6 if few else 1.6e-3)}
    if kind in ("step", "moe_step"):
        return {"rel": 6e-6}   # seen: 1.4e-6, 5e-7 (the sums' common part outweighs the rounding)
    if kind == "selected":
        return {"rel": 2e-4}   # seen: 8e-8 on equal Q8_1 blocks
    if kind == "matmul":
        return {"rel": 1e-2}   # bf16 weights and activations (seen: 2.4e-3)
    return {"rel": 1e-3}       # moe: bf16 weights, activations and hidden vectors (seen: 1.7e-4)
