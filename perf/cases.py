"""The calls a user of this package makes, as cases to be timed: triangle attention, the triangle multiplicative
update, attention with pair bias, and the pair stack built from them.

``listed()`` gives a handful of them, ``draw()`` more of the same ranges.  Every case goes through the package's public
functions on tensors that are on the GPU already, as inside a model; training cases take the gradients of every
differentiable input for a given upstream gradient.
"""

import math

import torch

from geometric_nn_ops_b200 import pairstack
from geometric_nn_ops_b200.triangle import attention_pair_bias, triangle_attention, triangle_multiplicative_update

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}


def _attention(name, n, mode, dtype="bf16", precision="ieee", layout="native", heads=4, dim=32):
    return {"name": name, "op": "attention", "n": n, "mode": mode, "dtype": dtype, "precision": precision, "layout": layout,
            "heads": heads, "dim": dim}


def _trimul(name, n, mode, direction, dtype="bf16", precision="ieee", c=128):
    return {"name": name, "op": "trimul", "n": n, "mode": mode, "direction": direction, "dtype": dtype,
            "precision": precision, "c": c}


def _pair_bias(name, n, samples, dtype="bf16", heads=16, dim=48):
    return {"name": name, "op": "pair_bias", "n": n, "samples": samples, "dtype": dtype, "heads": heads, "dim": dim}


def _stack(name, n, blocks, dtype="bf16"):
    return {"name": name, "op": "stack", "n": n, "blocks": blocks, "dtype": dtype}


def listed():
    return [
        # A short peptide, one inference call: launches and host work are most of it.
        _attention("attn_infer_n64", 64, "infer"),
        # Inference on a mid-sized chain through the cuequivariance (B, N, H, S, D) layout, a transposed view.
        _attention("attn_infer_n256_cueq", 256, "infer", layout="cueq"),
        # A chain at its own length: sequence lengths are seldom a multiple of eight.
        _attention("attn_train_n301", 301, "train"),
        # Fine-tuning in fp32 with the TF32 switch on.
        _attention("attn_train_n256_tf32", 256, "train", dtype="fp32", precision="tf32"),
        # The training step of the large crop, the benchmark's attention.
        _attention("attn_train_n768", 768, "train"),
        # fp32 inference at torch's default precision on a small pair tensor.
        _trimul("trimul_infer_n64_fp32", 64, "infer", "outgoing", dtype="fp32"),
        # Inference on a chain at its own length.
        _trimul("trimul_infer_n203", 203, "infer", "incoming"),
        # The training step of the usual crop.
        _trimul("trimul_train_n384", 384, "train", "incoming"),
        # The fp32 variant of training, with the TF32 switch on.
        _trimul("trimul_train_n512_tf32", 512, "train", "outgoing", dtype="fp32", precision="tf32"),
        # The training step of the large crop, the benchmark's multiplicative update.
        _trimul("trimul_train_n768", 768, "train", "outgoing"),
        # Single-track attention of a pairformer block: one row of tokens, many heads, bias projected from the pairs.
        _pair_bias("pair_bias_n384", 384, 1),
        # Whole-complex inference: four blocks of the pair stack.
        _stack("stack_infer_n1024", 1024, 4),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi, ragged_hi):
    """A padded length (a multiple of eight) up to ``hi`` or any length up to ``ragged_hi``, in equal parts."""
    if rng.random() < 0.5:
        return max(8, (_log_uniform(rng, lo, hi) + 7) // 8 * 8)
    return _log_uniform(rng, lo, ragged_hi)


def draw(rng):
    op = rng.choice(["attention"] * 4 + ["trimul"] * 4 + ["pair_bias"] * 2 + ["stack"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])
    precision = rng.choice(["ieee", "tf32"]) if dtype == "fp32" else "ieee"
    mode = rng.choice(["infer", "train"])
    # fp32 and ragged lengths stay where one draw costs no more than the largest listed case
    if op == "attention":
        n = _length(rng, 48, 768, 448) if dtype != "fp32" else _length(rng, 48, 384, 384)
        heads, dim = rng.choice([(4, 32), (4, 32), (8, 32), (4, 64)])
        case = _attention("", n, mode, dtype, precision, rng.choice(["native", "cueq"]), heads, dim)
    elif op == "trimul":
        wide = dtype != "fp32" or precision == "tf32"
        n = _length(rng, 48, 768, 448) if wide else _length(rng, 48, 384, 384)
        case = _trimul("", n, mode, rng.choice(["outgoing", "incoming"]), dtype, precision)
    elif op == "pair_bias":
        case = _pair_bias("", _length(rng, 64, 1024, 1024), rng.randint(1, 4), "bf16" if dtype == "fp32" else dtype)
    else:
        case = _stack("", _length(rng, 64, 1024, 288), rng.randint(1, 4))
    del case["name"]
    return case


# --------------------------------------------------------------------------------------------------- inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _attention_inputs(case, seed):
    g, dt = _generator(seed), DTYPES[case["dtype"]]
    n, h, d = case["n"], case["heads"], case["dim"]
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dt)  # noqa: E731
    if case["layout"] == "cueq":     # stored [B, N, H, S, D], handed over as a view
        token = lambda: rn(1, n, h, n, d).transpose(2, 3)  # noqa: E731
    else:
        token = lambda: rn(1, n, n, h, d)  # noqa: E731
    q, k, v, d_out = token(), token(), token(), token()
    bias = rn(1, 1, h, n, n)
    mask = torch.rand(1, n, 1, 1, n, generator=g, device="cuda") < 0.95
    mask[..., 0] = True
    state = {"case": case, "q": q, "k": k, "v": v, "bias": bias, "mask": mask}
    if case["mode"] == "train":
        for name in ("q", "k", "v", "bias"):
            state[name].requires_grad_()
        state["d_out"] = d_out
    return state


def _trimul_inputs(case, seed):
    g, dt = _generator(seed), DTYPES[case["dtype"]]
    n, c = case["n"], case["c"]
    rn = lambda *s, sc=1.0: torch.randn(*s, generator=g, device="cuda") * sc  # noqa: E731
    x = rn(1, n, n, c).to(dt)
    mask = (torch.rand(1, n, n, generator=g, device="cuda") < 0.9).to(dt)
    w = {"norm_in_weight": 1 + rn(c, sc=0.02), "norm_in_bias": rn(c, sc=0.02),
         "p_in_weight": rn(2 * c, c, sc=c ** -0.5), "g_in_weight": rn(2 * c, c, sc=c ** -0.5),
         "norm_out_weight": 1 + rn(c, sc=0.02), "norm_out_bias": rn(c, sc=0.02),
         "p_out_weight": rn(c, c, sc=c ** -0.5), "g_out_weight": rn(c, c, sc=c ** -0.5)}
    w = {k: t.to(dt) for k, t in w.items()}
    state = {"case": case, "x": x, "mask": mask, "w": w}
    if case["mode"] == "train":
        x.requires_grad_()
        for t in w.values():
            t.requires_grad_()
        state["d_out"] = rn(1, n, n, c).to(dt)
    return state


def _pair_bias_inputs(case, seed):
    g, dt = _generator(seed), DTYPES[case["dtype"]]
    n, m, h, d = case["n"], case["samples"], case["heads"], case["dim"]
    width, zc = h * d, 128
    rn = lambda *s, sc=1.0: (torch.randn(*s, generator=g, device="cuda") * sc).to(dt)  # noqa: E731
    mask = torch.ones(1, n, device="cuda", dtype=dt)
    mask[:, n - n // 16:] = 0
    return {"case": case, "s": rn(m, n, width), "q": rn(m, h, n, d), "k": rn(m, h, n, d), "v": rn(m, h, n, d),
            "z": rn(1, n, n, zc), "mask": mask,
            "w": {"proj_g_weight": rn(width, width, sc=width ** -0.5), "proj_o_weight": rn(width, width, sc=width ** -0.5),
                  "proj_z_weight": rn(h, zc, sc=zc ** -0.5), "ln_z_weight": rn(zc, sc=0.02) + 1}}


def _stack_inputs(case, seed):
    dt, n = DTYPES[case["dtype"]], case["n"]
    z = torch.randn(1, n, n, 128, generator=_generator(seed), device="cuda").to(dt)
    residues = torch.ones(n, device="cuda")
    residues[n - n // 16:] = 0       # the padded tail of the complex
    mask = (residues[:, None] * residues[None, :]).reshape(1, n, n).to(dt)
    blocks = [pairstack.make_block_weights(1000 * seed + i, dtype=dt, device="cuda") for i in range(case["blocks"])]
    return {"case": case, "z": z, "mask": mask, "blocks": blocks}


def prepare(case, seed):
    # the process-wide switch a program sets once
    torch.backends.cuda.matmul.fp32_precision = case.get("precision", "ieee")
    return {"attention": _attention_inputs, "trimul": _trimul_inputs, "pair_bias": _pair_bias_inputs,
            "stack": _stack_inputs}[case["op"]](case, seed)


# ----------------------------------------------------------------------------------------------------- a pass

def _run_attention(st):
    if st["case"]["mode"] == "infer":
        with torch.no_grad():
            return triangle_attention(st["q"], st["k"], st["v"], st["bias"], st["mask"])
    leaves = [st["q"], st["k"], st["v"], st["bias"]]
    out = triangle_attention(*leaves, st["mask"])
    return (out.detach(), *torch.autograd.grad(out, leaves, grad_outputs=st["d_out"]))


def _run_trimul(st):
    direction, w = st["case"]["direction"], st["w"]
    if st["case"]["mode"] == "infer":
        with torch.no_grad():
            return triangle_multiplicative_update(st["x"], direction, st["mask"], **w)
    out = triangle_multiplicative_update(st["x"], direction, st["mask"], **w)
    return (out.detach(), *torch.autograd.grad(out, [st["x"], *w.values()], grad_outputs=st["d_out"]))


def _run_pair_bias(st):
    with torch.no_grad():
        return attention_pair_bias(st["s"], st["q"], st["k"], st["v"], st["z"], mask=st["mask"], **st["w"])[0]


def _run_stack(st):
    return pairstack.pair_stack(st["z"], st["mask"], st["blocks"])


def run(state):
    return {"attention": _run_attention, "trimul": _run_trimul, "pair_bias": _run_pair_bias,
            "stack": _run_stack}[state["case"]["op"]](state)


# ------------------------------------------------------------------------------------ what a pass cannot do without

def work(case):
    n, e = case["n"], BYTES[case["dtype"]]
    if case["op"] == "attention":
        tensor, plane = n * n * case["heads"] * case["dim"] * e, case["heads"] * n * n * e
        core = n ** 3 * case["heads"] * case["dim"]
        if case["mode"] == "infer":
            return {"bytes": 4 * tensor + plane + n * n, "flops": 4 * core}
        return {"bytes": 8 * tensor + 2 * plane + n * n, "flops": 14 * core}
    if case["op"] == "trimul":
        c = case["c"]
        pairs, weights = n * n * c * e, (6 * c * c + 4 * c) * e
        flops = 2 * n * n * c * 6 * c + 2 * n ** 3 * c
        if case["mode"] == "infer":
            return {"bytes": 2 * pairs + n * n * e + weights, "flops": flops}
        return {"bytes": 4 * pairs + n * n * e + 2 * weights, "flops": 3 * flops}
    if case["op"] == "pair_bias":
        m, width, zc = case["samples"], case["heads"] * case["dim"], 128
        flops = 4 * m * n * n * width + 4 * m * n * width * width + 2 * n * n * zc * case["heads"]
        return {"bytes": (n * n * zc + 5 * m * n * width + 2 * width * width) * e, "flops": flops}
    c = 128
    block_weights = 2 * (6 * c * c + 4 * c) + 2 * (3 * c * c + 4 * c)
    return {"bytes": (2 * n * n * c + n * n + case["blocks"] * block_weights) * e,
            "flops": pairstack.stack_flops(n, case["blocks"], c)}


def tolerance(case):
    if case["dtype"] == "fp32":      # sums of 1e2 to 1e5 terms in another order; TF32 keeps ten bits of each factor
        return {"rel": 2e-3 if case["precision"] == "tf32" else 2e-5}
    if case["op"] == "stack":        # sixteen residual updates, each rounded to bf16
        return {"rel": 2e-2}
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 4e-3}
