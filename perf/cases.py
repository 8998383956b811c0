"""Workloads for timing the framework through its front end, `i_b200.ilang`.

A case is a plain dict.  `listed()` names the standing ones, `draw(rng)` gives another of the same
ranges, `prepare` makes what a program has in hand before the call (the tensors, the output it reuses
and the compiled component), and `run` makes the one call.  `work` and `tolerance` say what a call
cannot do without and how far two correct implementations of its arithmetic lie apart.

Three ways of calling are in use: `into` writes CUDA outputs the caller keeps (a loop), `exec` returns
new CUDA tensors (`exec_torch`), `host` hands over NumPy arrays and gets NumPy arrays (`exec_numpy`).
"""
import functools
import math

import torch

from i_b200 import ilang

i, I = ilang.i, ilang.I


# ---- components -------------------------------------------------------------------------------
# A program builds its components once and calls them many times; so does this file.

@functools.lru_cache(maxsize=None)
def attention(batched, scaled, fused, precision):
    """The README's attention component.  `batched`: a leading head axis.  `scaled`: 1/sqrt(d) as a
    scalar input on the logits.  Not `fused`: the schedule of the reference's test scripts, which
    keeps the contractions and the softmax as steps of their own."""
    h = "h" if batched else ""
    stage = "0" if fused else ""
    mm_t = i(f"{h}ik*{h}jk~{h}ijk | i:16,j:16 | {h}jii'j'k") >> i(f"+{h}ijk~{h}ij | i:16,j:16 | {h}jii'j'k0")

    def rows(op, unary):
        """`I & fold`, then the map that reads both: the two halves around the exponential."""
        if fused:
            return (I & i(f"{op}{h}ij~{h}i | i:16,j:16 | {h}ji0i'j'")) >> i(f"{h}ij{unary}{h}i~{h}ij | i:16,j:16 | {h}ji01i'j'")
        return (I & i(f"{op}{h}ij~{h}i | i:16,j:16 | {h}jii'j'")) >> i(f"{h}ij{unary}{h}i~{h}ij | i:16,j:16 | {h}1jii'j'")

    exp = i(f"^{h}ij~{h}ij | i:16,j:16 | {h}ji{stage}i'j'")
    mm = i(f"{h}ij*{h}jk~{h}ikj | i:16,j:16 | {h}ji{stage}i'kj'") >> i(f"+{h}ikj~{h}ik | i:16,j:16 | {h}jii'kj'0")
    logits = mm_t
    if scaled:
        logits = (mm_t | I) >> i(f"{h}ij*.~{h}ij | i:16,j:16 | {h}ji{stage}i'j'")
    return (logits >> rows(">", "-") >> exp >> rows("+", "/") >> mm).set_precision(precision)


@functools.lru_cache(maxsize=None)
def contraction(batched, layout, layer, precision):
    """C = A B over k, either operand stored with k last ("n" for A, "t" for B as in a transposed
    second operand) or first.  `layer`: with a bias per column and a rectifier on the result."""
    b = "b" if batched else ""
    left = f"{b}ik" if layout[0] == "n" else f"{b}ki"
    right = f"{b}jk" if layout[1] == "t" else f"{b}kj"
    c = i(f"{left}*{right}~{b}ijk") >> i(f"+{b}ijk~{b}ij")
    if layer:
        c = c >> i(f"{b}ij+j~{b}ij") >> i(f">{b}ij~{b}ij")
    return c.set_precision(precision)


@functools.lru_cache(maxsize=None)
def other(which):
    """The components without a precision choice: softmax, log-sum-exp, maps, folds, the MLP."""
    shift = (I & i(">ij~i")) >> i("ij-i~ij")
    return {
        "softmax": lambda: shift >> i("^ij~ij") >> ((I & i("+ij~i")) >> i("ij/i~ij")),
        "logsumexp": lambda: (I & i(">ij~i")) >> (i("ij-i~ij") >> i("^ij~ij") >> i("+ij~i") >> i("$i~i")),
        "exp": lambda: i("^ij~ij"),
        "gate": lambda: i("ij+j~ij") >> i(">ij~ij") >> i("ij*ij~ij"),
        "shift_exp_div": lambda: i("ij-i~ij") >> i("^ij~ij") >> i("ij/i~ij"),
        "transpose": lambda: i("ij~ji"),
        "sum_rows": lambda: i("+ij~i"),
        "max_rows": lambda: i(">ij~i"),
        "sum_columns": lambda: i("+ij~j"),
        "max_columns": lambda: i(">ij~j"),
        "sum_all": lambda: i("+ij~."),
        "mlp": lambda: (I | (i("ij*j~ij") >> i("+ij~i") >> i(">i~i"))) >> (i("ij*j~ij") >> i("+ij~i")),
    }[which]()


MAPS = ("exp", "gate", "shift_exp_div", "transpose")
FOLDS = ("sum_rows", "max_rows", "sum_columns", "max_columns", "sum_all")


# ---- cases ------------------------------------------------------------------------------------

def attention_case(heads, nq, nk, d, dv=None, precision="auto", scaled=False, fused=True, call="into"):
    return {"kind": "attention", "heads": heads, "nq": nq, "nk": nk, "d": d, "dv": d if dv is None else dv,
            "precision": precision, "scaled": scaled, "fused": fused, "call": call}


def contract_case(m, n, k, batch=1, layout="nt", layer=False, precision="auto", call="into"):
    return {"kind": "contract", "m": m, "n": n, "k": k, "batch": batch, "layout": layout, "layer": layer,
            "precision": precision, "call": call}


def other_case(which, rows, cols, call="into", **more):
    return {"kind": which, "rows": rows, "cols": cols, "call": call, **more}


def listed():
    named = {
        # The README's demo: one small head on the GPU, a new output each time.  Latency.
        "attention_128_d64": attention_case(1, 128, 128, 64, call="exec"),
        # The reference's flash-attn.py as it is called there: NumPy in, NumPy out, d = 2048.
        "attention_host_32_d2048": attention_case(1, 32, 32, 2048, call="host"),
        # The headline: one long head.
        "attention_16384_d128": attention_case(1, 16384, 16384, 128),
        # A batch of short sequences, one call for all heads (prefill).
        "attention_64x2048_d128": attention_case(64, 2048, 2048, 128),
        # One new query per head against a fixed context of a length that divides nothing (decode).
        "attention_decode_32x10000": attention_case(32, 1, 10000, 128),
        # The opt-in bf16 arithmetic, 1/sqrt(d) in the component, ragged lengths, small heads.
        "attention_bf16_6x1500_d64": attention_case(6, 1500, 2300, 64, precision="bf16", scaled=True),
        # Row softmax of the reference's second configuration.
        "softmax_8192x8192": other_case("softmax", 8192, 8192),
        # The contraction of its third.
        "mm_t_8192x8192x4096": contract_case(8192, 8192, 4096),
        # A layer of an ordinary network: product, bias, rectifier; the weights stored k first.
        "layer_1000x3000x700": contract_case(1000, 3000, 700, layout="nn", layer=True),
        # A caller who asks for fp32 arithmetic, at a depth no tile divides.
        "mm_fp32_1024x1000x1001": contract_case(1024, 1000, 1001, layout="nn", precision="fp32"),
        # A fold, a chain of maps under a fold, a map: the memory-bound side in one program.
        "logsumexp_8192x8192": other_case("logsumexp", 8192, 8192),
        # One vector through a two-layer network (the reference's test.py), latency and bandwidth.
        "mlp_4096x2048": other_case("mlp", 4096, 2048, outs=1000, call="exec"),
    }
    return [dict(case, name=name) for name, case in named.items()]


def extent(rng, lo, hi):
    """A size between lo and hi, spread over the logarithm; half of them multiples of 64 or 8."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    unit = rng.choice((1, 1, 8, 64))
    return max(lo, min(hi, n // unit * unit if n >= 2 * unit else n))


MOST_FLOP = 1.3e11         # a drawn case stays below the long head ...
MOST_FP32_FLOP = 3e9       # ... and in time where the arithmetic may be fp32
MOST_VALUES = 6.7e7        # values of the largest array
MOST_SCORES = 2e7          # values of a score matrix that goes through memory
MOST_HOST_VALUES = 4e6


def draw(rng):
    while True:
        case = draw_any(rng)
        cost = work(case)
        slow = case["kind"] in ("attention", "contract") and (arithmetic(case) == "fp32" or case.get("k", 0) % 4)
        values = cost["bytes"] / 4
        if cost["flops"] > (MOST_FP32_FLOP if slow else MOST_FLOP) or values > 2 * MOST_VALUES:
            continue
        if case["kind"] == "attention" and not case["fused"] and case["heads"] * case["nq"] * case["nk"] > MOST_SCORES:
            continue
        if case["call"] == "host" and values > MOST_HOST_VALUES:
            continue
        return case


def draw_any(rng):
    call = rng.choice(("into", "into", "into", "exec", "host"))
    kind = rng.choice(("attention", "attention", "attention", "decode", "contract", "contract", "contract",
                       "softmax", "logsumexp", "map", "fold", "mlp"))
    if kind == "attention":
        d = rng.choice((32, 64, 80, 128, 128))
        return attention_case(extent(rng, 1, 64), extent(rng, 16, 16384), extent(rng, 16, 16384), d,
                              dv=rng.choice((d, d, 48)),
                              precision=rng.choice(("auto", "auto", "auto", "tf32", "tf32_f16", "bf16", "fp32")),
                              scaled=rng.random() < 0.3, fused=rng.random() < 0.8, call=call)
    if kind == "decode":
        return attention_case(extent(rng, 8, 64), extent(rng, 1, 16), extent(rng, 512, 16384),
                              rng.choice((64, 128)), scaled=rng.random() < 0.3, call=call)
    if kind == "contract":
        return contract_case(extent(rng, 8, 8192), extent(rng, 8, 8192), extent(rng, 16, 8192),
                             batch=rng.choice((1, 1, 1, extent(rng, 2, 32))),
                             layout=rng.choice(("nt", "nt", "nn", "nn", "tn")), layer=rng.random() < 0.4,
                             precision=rng.choice(("auto", "auto", "auto", "tf32", "f16", "bf16", "fp32")), call=call)
    if kind == "mlp":
        return other_case("mlp", extent(rng, 64, 8192), extent(rng, 64, 8192), outs=extent(rng, 8, 4096), call=call)
    which = {"map": rng.choice(MAPS), "fold": rng.choice(FOLDS)}.get(kind, kind)
    return other_case(which, extent(rng, 8, 16384), extent(rng, 16, 65536), call=call)


def arithmetic(case):
    """What the contractions of a case compute in: "fp32", "10 bits" (TF32's mantissa) or "bf16".
    Unasked, products below 2^28 FLOP, and plain contractions over a depth that is not a multiple of
    four, are fp32."""
    asked = case.get("precision", "fp32")
    if asked == "auto":
        if case["kind"] == "contract":
            small = 2 * case["batch"] * case["m"] * case["n"] * case["k"] < 2 ** 28 or case["k"] % 4 != 0
        else:
            # Fused, the two contractions decide together; as steps of their own, each for itself.
            depth = 2 * case["d"] if case["fused"] else max(case["d"], case["dv"])
            small = 2 * case["heads"] * case["nq"] * case["nk"] * depth < 2 ** 28
        return "fp32" if small else "10 bits"
    return asked if asked in ("fp32", "bf16") else "10 bits"


def shapes(case):
    """Shapes of the inputs in the component's order, then of the output."""
    kind = case["kind"]
    if kind == "attention":
        h = (case["heads"],) if case["heads"] > 1 else ()
        q, k, v = h + (case["nq"], case["d"]), h + (case["nk"], case["d"]), h + (case["nk"], case["dv"])
        return ([q, k, (), v] if case["scaled"] else [q, k, v]), h + (case["nq"], case["dv"])
    if kind == "contract":
        b = (case["batch"],) if case["batch"] > 1 else ()
        m, n, k = case["m"], case["n"], case["k"]
        left = b + ((m, k) if case["layout"][0] == "n" else (k, m))
        right = b + ((n, k) if case["layout"][1] == "t" else (k, n))
        return [left, right] + ([(n,)] if case["layer"] else []), b + (m, n)
    r, c = case["rows"], case["cols"]
    if kind == "mlp":
        return [(case["outs"], r), (r, c), (c,)], (case["outs"],)
    ins = {"gate": [(r, c), (c,), (r, c)], "shift_exp_div": [(r, c), (r,), (r,)]}.get(kind, [(r, c)])
    out = {"transpose": (c, r), "sum_columns": (c,), "max_columns": (c,), "sum_all": ()}.get(
        kind, (r,) if kind in ("sum_rows", "max_rows", "logsumexp") else (r, c))
    return ins, out


def component(case):
    if case["kind"] == "attention":
        return attention(case["heads"] > 1, case["scaled"], case["fused"], case["precision"])
    if case["kind"] == "contract":
        return contraction(case["batch"] > 1, case["layout"], case["layer"], case["precision"])
    return other(case["kind"])


def prepare(case, seed):
    """Standard normal values scaled as the path meets them: queries by 1/sqrt(d) (or that factor as
    an input), operands of a product uniform in (-1, 1), logits N(0, 4), weights by 1/sqrt(fan-in)."""
    made, out = shapes(case)
    kind = case["kind"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def normal(shape, scale=1.0):
        return torch.randn(shape, device="cuda", generator=g).mul_(scale)

    def uniform(shape, low):
        return torch.rand(shape, device="cuda", generator=g).mul_(1.0 - low).add_(low)

    if kind == "attention":
        factor = case["d"] ** -0.5
        inputs = [normal(s) for s in made]
        if case["scaled"]:
            inputs[2] = torch.tensor(factor, device="cuda")
        else:
            inputs[0] *= factor
    elif kind == "contract":
        inputs = [uniform(s, -1.0) for s in made]
    elif kind == "mlp":
        inputs = [normal(made[0], made[0][1] ** -0.5), normal(made[1], made[1][1] ** -0.5), normal(made[2])]
    elif kind == "shift_exp_div":
        inputs = [normal(made[0], 2.0), normal(made[1]).abs_().add_(2.0), uniform(made[2], 0.5)]
    elif kind in FOLDS:
        inputs = [uniform(s, 0.0) for s in made]
    else:
        inputs = [normal(s, 2.0) for s in made]
    if case["call"] == "host":
        inputs = [x.cpu().numpy() for x in inputs]
    state = {"component": component(case), "call": case["call"], "inputs": inputs}
    if case["call"] == "into":
        state["out"] = torch.empty(out, device="cuda")
    return state


def run(state):
    f, inputs = state["component"], state["inputs"]
    if state["call"] == "into":
        return f.into(state["out"], *inputs)
    return f.exec_torch(*inputs) if state["call"] == "exec" else f.exec_numpy(*inputs)


def work(case):
    """Every input read once and the output written once, four bytes each; a multiply and an add per
    term of a product, and otherwise one operation per value and operator."""
    made, out = shapes(case)
    sizes = [math.prod(s) for s in made + [out]]
    kind = case["kind"]
    if kind == "attention":
        flops = 2 * case["heads"] * case["nq"] * case["nk"] * (case["d"] + case["dv"])
    elif kind == "contract":
        flops = 2 * case["batch"] * case["m"] * case["n"] * case["k"]
    elif kind == "mlp":
        flops = 2 * (sizes[0] + sizes[1])
    else:
        flops = {"softmax": 5, "logsumexp": 4, "gate": 3, "shift_exp_div": 3, "transpose": 0}.get(kind, 1) * sizes[0]
    return {"bytes": 4 * sum(sizes), "flops": flops}


def tolerance(case):
    """Operands with ten mantissa bits carry 2^-11 to 2^-10 each, bf16's seven eight times that; fp32
    sums differ by their order."""
    return {"rel": {"fp32": 1e-5, "10 bits": 3e-3, "bf16": 1e-2}[arithmetic(case)]}
