"""triangle_multiplicative_update on the GPU against the oracle, golden fixtures and known answers.

Structural cases mirror the reference's tests/test_trimul.py (zero mask :70-90, biases matter
:93-113, directions differ :116-131, bad direction :134-148, mask=None == ones :151-164,
broadcast mask :167-182, tf32 != ieee :185-201, accuracy :208-250, batched :253-272, widths
:305-341, LayerNorm weights :344-382).
"""

import glob
import os

import numpy as np
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

GOLD = sorted(glob.glob(os.path.join(os.path.dirname(__file__), "golden", "trimul_*.npz")))


@pytest.fixture(scope="module")
def tmu():
    from geometric_nn_ops_b200.triangle import trimul_b200
    return trimul_b200


def _tol(dtype, precision):
    cos_min, fro = util.TRIMUL_TOL[dtype, precision]
    if dtype == torch.float32 and precision == "ieee":
        return cos_min, util.IEEE_REL_FRO, util.MAX_ABS_REL["ieee32"]
    if dtype == torch.float32:
        return cos_min, fro, util.MAX_ABS_REL["tf32"]
    return cos_min, fro, util.MAX_ABS_REL[dtype]


@pytest.mark.parametrize("path", GOLD, ids=[os.path.basename(p) for p in GOLD])
def test_golden_fp32_ieee(tmu, path):
    g = dict(np.load(path))
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    w = {k[2:]: dev(v) for k, v in g.items() if k.startswith("w_")}
    mask = dev(g["mask"]) if "mask" in g else None
    with util.matmul_precision("ieee"):
        out, grads = util.trimul_fwd_bwd(tmu, dev(g["x"]), mask, w, str(g["direction"]), dev(g["d_out"]))
    util.check_close("out", out, g["out"], 1 - 1e-9, util.IEEE_REL_FRO, 1e-4)
    for name, val in grads.items():
        util.check_close("grad_" + name, val, g["grad_" + name], 1 - 1e-9, util.IEEE_REL_FRO, 1e-4)


CASES = [  # B, N, C, Ch, biases
    (1, 32, 128, 128, False), (2, 17, 64, 32, True), (1, 40, 96, 96, False), (1, 24, 256, 128, True),
    (1, 128, 128, 128, False),
    # 128 channels with a ragged last tile (1600 = 12 * 128 + 64 pixels) and projection biases; two batch entries
    # (the fused input kernel across a plane boundary inside a tile, the two-kernel output path)
    (1, 40, 128, 128, True), (2, 24, 128, 128, True),
]
MODES = [(torch.float32, "ieee"), (torch.float32, "tf32"), (torch.bfloat16, "ieee"), (torch.float16, "ieee")]


@pytest.mark.parametrize("direction", ["outgoing", "incoming"])
@pytest.mark.parametrize("case", CASES, ids=str)
@pytest.mark.parametrize("dtype,precision", MODES, ids=lambda v: str(v).replace("torch.", ""))
def test_oracle_fwd_bwd(tmu, case, dtype, precision, direction):
    B, N, C, Ch, biases = case
    x, mask, w, d_out = util.trimul_inputs(B, N, C, Ch, dtype, seed=N + C, biases=biases)
    with util.matmul_precision(precision):
        out, grads = util.trimul_fwd_bwd(tmu, x, mask, w, direction, d_out)
    from geometric_nn_ops_b200 import _lib
    tensor_core = C == 128 and Ch == 128 and N % 8 == 0 and not (dtype == torch.float32 and precision == "ieee")
    assert _lib.last_path() == ("tcgen05" if tensor_core else "simt")
    o_ref, g_ref = util.trimul_oracle(x, mask, w, direction, d_out)
    cos_min, fro, mar = _tol(dtype, precision)
    util.check_close("out", out, o_ref, cos_min, fro, mar)
    for name, val in grads.items():
        util.check_close("grad_" + name, val, g_ref[name], cos_min, fro, mar)


def test_baseline_config0_forward(tmu):
    """outgoing, fp32 (default precision = ieee), N=64, C=Ch=128, forward only."""
    x, mask, w, _ = util.trimul_inputs(1, 64, 128, 128, torch.float32, seed=0)
    with torch.no_grad():
        out = tmu(x, "outgoing", mask, **w)
    o_ref = util.trimul_oracle(x, mask, w, "outgoing", torch.zeros_like(x))[0]
    util.check_close("out", out, o_ref, 1 - 1e-9, util.IEEE_REL_FRO, 1e-4)


def test_structure(tmu):
    x, mask, w, _ = util.trimul_inputs(2, 20, 32, 16, torch.float32, seed=1, biases=True)
    with torch.no_grad():
        base = tmu(x, "outgoing", mask, **w)
        assert torch.equal(tmu(x, "outgoing", mask, **w), base)  # deterministic
        assert not torch.equal(tmu(x, "incoming", mask, **w), base)
        # all-zero mask: the contraction output is zero, the output depends on z only through the gate
        zero = tmu(x, "outgoing", torch.zeros_like(mask), **w)
        u0 = w["norm_out_bias"].float() @ w["p_out_weight"].float().T + w["p_out_bias"].float()
        z = torch.nn.functional.layer_norm(x, (32,), w["norm_in_weight"], w["norm_in_bias"], 1e-5)
        gate = torch.sigmoid(z @ w["g_out_weight"].T + w["g_out_bias"])
        assert (zero - u0 * gate).abs().max() < 1e-5
        # mask=None equals a mask of ones; a broadcast mask equals its expansion
        assert torch.equal(tmu(x, "outgoing", None, **w), tmu(x, "outgoing", torch.ones_like(mask), **w))
        assert torch.equal(tmu(x, "incoming", mask[0], **w), tmu(x, "incoming", mask[:1].expand(2, -1, -1), **w))
        # every projection bias matters
        for name in ("p_in_bias", "g_in_bias", "p_out_bias", "g_out_bias"):
            w2 = dict(w, **{name: w[name] + 0.5})
            assert not torch.equal(tmu(x, "outgoing", mask, **w2), base), name
        # batch entries are independent
        assert torch.equal(tmu(x[1:], "outgoing", mask[1:], **w), base[1:])
    with pytest.raises(ValueError, match="direction must be one of"):
        tmu(x, "sideways", mask, **w)


def test_public_wrapper_and_dtypes():
    from geometric_nn_ops_b200.triangle import triangle_multiplicative_update as op
    x, mask, w, _ = util.trimul_inputs(1, 12, 32, 16, torch.float32, seed=2)
    out = op(x, "incoming", mask, **w)
    assert out.shape == x.shape and out.dtype == x.dtype
    # 5-D input (two leading dims)
    o5 = op(x.reshape(1, 1, 12, 12, 32), "incoming", mask.reshape(1, 1, 12, 12), **w)
    assert torch.equal(o5.reshape(out.shape), out)
    o64 = op(x.double(), "incoming", mask.double(), **{k: v.double() for k, v in w.items()})
    assert o64.dtype == torch.float64 and torch.equal(o64.float(), out)


def test_tf32_differs_from_ieee(tmu):
    x, mask, w, d_out = util.trimul_inputs(1, 32, 64, 64, torch.float32, seed=3)
    with util.matmul_precision("ieee"):
        o1, g1 = util.trimul_fwd_bwd(tmu, x, mask, w, "outgoing", d_out)
    with util.matmul_precision("tf32"):
        o2, g2 = util.trimul_fwd_bwd(tmu, x, mask, w, "outgoing", d_out)
    assert not torch.equal(o1, o2)
    assert not torch.equal(g1["x"], g2["x"])


@pytest.mark.parametrize("gamma", ["zero", "tiny"])
def test_layernorm_weight_edge_cases(tmu, gamma):
    x, mask, w, d_out = util.trimul_inputs(1, 16, 64, 64, torch.float32, seed=4)
    val = 0.0 if gamma == "zero" else 1e-6
    w = dict(w, norm_in_weight=torch.full_like(w["norm_in_weight"], val),
             norm_out_weight=torch.full_like(w["norm_out_weight"], val))
    out, grads = util.trimul_fwd_bwd(tmu, x, mask, w, "outgoing", d_out)
    o_ref, g_ref = util.trimul_oracle(x, mask, w, "outgoing", d_out)
    util.check_close("out", out, o_ref, 1 - 1e-6, 1e-4)
    for name in ("x", "norm_in_bias", "p_out_weight"):
        util.check_close("grad_" + name, grads[name], g_ref[name], 1 - 1e-6, 1e-3)


@pytest.mark.parametrize("direction", ["outgoing", "incoming"])
def test_headline_size_properties(tmu, direction):
    """N=768, C=128 bf16: finite, deterministic, batch-independent sub-problem check via linearity in d_out."""
    x, mask, w, d_out = util.trimul_inputs(1, 768, 128, 128, torch.bfloat16, seed=5)
    out, g1 = util.trimul_fwd_bwd(tmu, x, mask, w, direction, d_out)
    from geometric_nn_ops_b200 import _lib
    assert _lib.last_path() == "tcgen05"
    assert torch.isfinite(out.float()).all()
    _, g2 = util.trimul_fwd_bwd(tmu, x, mask, w, direction, 2 * d_out)
    for name in g1:
        a, b = g1[name].float(), g2[name].float()
        assert torch.isfinite(a).all(), name
        rel = (2 * a - b).norm() / b.norm().clamp_min(1e-20)
        assert rel < 2e-2, (name, float(rel))


# ---- the tensor-core path at sizes with several N tiles and a multi-step K loop, against the fp64 oracle ---------
@pytest.mark.parametrize("direction", ["outgoing", "incoming"])
@pytest.mark.parametrize("n", [256, 384])
@pytest.mark.parametrize("dtype,precision", [(torch.bfloat16, "ieee"), (torch.float32, "tf32")],
                         ids=lambda v: str(v).replace("torch.", ""))
def test_oracle_fwd_bwd_multi_tile(tmu, n, dtype, precision, direction):
    """BASELINE config 3's widths (C = C_hidden = 128, bf16 and fp32-tf32, both directions, forward + every
    gradient) at N=256 and N=384: 2-3 N tiles of 256/128 columns and 4-6 K blocks per contraction tile."""
    from geometric_nn_ops_b200 import _lib
    x, mask, w, d_out = util.trimul_inputs(1, n, 128, 128, dtype, seed=n)
    with util.matmul_precision(precision):
        out, grads = util.trimul_fwd_bwd(tmu, x, mask, w, direction, d_out)
    torch.cuda.synchronize()
    assert _lib.last_path() == "tcgen05"
    o_ref, g_ref = util.trimul_oracle(x, mask, w, direction, d_out)
    cos_min, fro, mar = _tol(dtype, precision)
    util.check_close("out", out, o_ref, cos_min, fro, mar)
    for name, val in grads.items():
        util.check_close("grad_" + name, val, g_ref[name], cos_min, fro, mar)


def _force_simt(on):
    if on:
        os.environ["TRI_B200_FORCE_SIMT"] = "1"
    else:
        os.environ.pop("TRI_B200_FORCE_SIMT", None)


@pytest.mark.parametrize("direction", ["outgoing", "incoming"])
@pytest.mark.parametrize("dtype,precision", [(torch.bfloat16, "ieee"), (torch.float32, "tf32")],
                         ids=lambda v: str(v).replace("torch.", ""))
def test_headline_size_against_exact_fp32_kernels(tmu, dtype, precision, direction):
    """BASELINE config 3 at its stated size (N=768): the tensor-core result against the exact-fp32 CUDA-core kernels
    on the same rounded inputs (those kernels are held to 1e-5 of the fp64 oracle by the cases above and the golden
    fixtures), forward and every gradient, within the reference's bf16 / tf32 tables."""
    from geometric_nn_ops_b200 import _lib
    x, mask, w, d_out = util.trimul_inputs(1, 768, 128, 128, dtype, seed=7)
    with util.matmul_precision(precision):
        out, grads = util.trimul_fwd_bwd(tmu, x, mask, w, direction, d_out)
    torch.cuda.synchronize()
    assert _lib.last_path() == "tcgen05"
    f = lambda t: None if t is None else t.float()  # noqa: E731
    _force_simt(True)
    try:
        with util.matmul_precision("ieee"):
            o_ref, g_ref = util.trimul_fwd_bwd(tmu, f(x), f(mask), {k: f(v) for k, v in w.items()}, direction, f(d_out))
        torch.cuda.synchronize()
        assert _lib.last_path() == "simt"
    finally:
        _force_simt(False)
    cos_min, fro, mar = _tol(dtype, precision)
    util.check_close("out", out, util.f64(o_ref), cos_min, fro, mar)
    for name, val in grads.items():
        util.check_close("grad_" + name, val, util.f64(g_ref[name]), cos_min, fro, mar)


def test_headline_size_pixels_against_oracle(tmu):
    """N=768 bf16 forward on a subset of output pixels against the fp64 oracle: out[i, j] only needs rows i and j
    (outgoing) of the projections, so the oracle runs on the sub-problem made of those rows."""
    n = 768
    x, mask, w, _ = util.trimul_inputs(1, n, 128, 128, torch.bfloat16, seed=8)
    with torch.no_grad():
        out = tmu(x, "outgoing", mask, **w)
    rows = [0, 5, 131, 400, 767]
    # sub-problem: x' = x[rows] as an R x N "pair" is not square; instead compute the oracle pieces directly
    from oracle import triangle_oracle as orc
    wn = {k: util.f64(v) for k, v in w.items()}
    xs, ms = util.f64(x)[0, rows], util.f64(mask)[0, rows]                  # [R, N, C], [R, N]
    z, _, _ = orc._layer_norm(xs, wn["norm_in_weight"], wn["norm_in_bias"], 1e-5)
    ab = orc._linear(z, wn["p_in_weight"], None) * orc._sigmoid(orc._linear(z, wn["g_in_weight"], None)) * ms[..., None]
    a, b = ab[..., :128], ab[..., 128:]
    t = np.einsum("ikc,jkc->ijc", a, b)                                      # [R, R, C]: pixels (rows[i], rows[j])
    u, _, _ = orc._layer_norm(t, wn["norm_out_weight"], wn["norm_out_bias"], 1e-5)
    zz = z[:, rows]                                                          # z at pixel (rows[i], rows[j])
    want = orc._linear(u, wn["p_out_weight"], None) * orc._sigmoid(orc._linear(zz, wn["g_out_weight"], None))
    got = out[0][rows][:, rows]
    cos_min, fro, mar = _tol(torch.bfloat16, "ieee")
    util.check_close("out", got, want, cos_min, fro, mar)


@pytest.mark.parametrize("n", [136, 264])
@pytest.mark.parametrize("dtype,precision", [(torch.bfloat16, "ieee"), (torch.float32, "tf32")], ids=lambda v: str(v).replace("torch.", ""))
def test_gate_gradients_from_reused_tiles(tmu, n, dtype, precision):
    """Several tiles per CTA, whose gradient buffers TMA fills again while the epilogue runs: the same bits on every pass."""
    x, mask, w, d_out = util.trimul_inputs(1, n, 128, 128, dtype, seed=n)
    with util.matmul_precision(precision):
        _, first = util.trimul_fwd_bwd(tmu, x, mask, w, "outgoing", d_out)
        for _ in range(8):
            _, again = util.trimul_fwd_bwd(tmu, x, mask, w, "outgoing", d_out)
            for name in first:
                assert torch.equal(again[name], first[name]), name


@pytest.mark.parametrize("name", ["mask", "p_in_weight", "norm_out_bias"])
def test_operands_on_another_device_are_refused(tmu, name):
    x, mask, w, _ = util.trimul_inputs(1, 16, 128, 128, torch.bfloat16, seed=1)
    if name == "mask":
        mask = mask.cpu()
    else:
        w[name] = w[name].cpu()
    with pytest.raises(ValueError, match=name):
        tmu(x, "outgoing", mask, **w)


@pytest.mark.parametrize("n", [8, 72, 104])
@pytest.mark.parametrize("dtype,precision", [m for m in MODES if m != (torch.float32, "ieee")], ids=lambda v: str(v).replace("torch.", ""))
def test_input_weight_gradients_over_few_tiles(tmu, n, dtype, precision):
    """The sums of the input gate's backward: one tile (fp32: two) for all CTAs, CTAs with one or two, and with two or three
    (fp32: three to five), so that every buffer is used, and not used, a second time."""
    x, mask, w, d_out = util.trimul_inputs(1, n, 128, 128, dtype, seed=n)
    with util.matmul_precision(precision):
        _, grads = util.trimul_fwd_bwd(tmu, x, mask, w, "outgoing", d_out)
    _, g_ref = util.trimul_oracle(x, mask, w, "outgoing", d_out)
    for name in ("x", "p_in_weight", "g_in_weight"):
        util.check_close("grad_" + name, grads[name], g_ref[name], *_tol(dtype, precision))


@pytest.mark.parametrize("frozen", [("p_in_weight", "g_in_weight"), ("p_in_weight",), ("g_in_weight",)], ids=lambda f: "+".join(n[0] for n in f))
@pytest.mark.parametrize("n", [8, 72, 104])
@pytest.mark.parametrize("dtype,precision", [m for m in MODES if m != (torch.float32, "ieee")], ids=lambda v: str(v).replace("torch.", ""))
def test_frozen_input_weights(tmu, n, dtype, precision, frozen):
    """The input gate's backward where no sums over the pixels are asked for, or those of one weight."""
    x, mask, w, d_out = util.trimul_inputs(1, n, 128, 128, dtype, seed=n, biases=True)
    leaves = {k: v.requires_grad_() for k, v in {"x": x, **w}.items() if k not in frozen}
    with util.matmul_precision(precision):
        out = tmu(x, "outgoing", mask, **w)
        grads = dict(zip(leaves, torch.autograd.grad(out, list(leaves.values()), grad_outputs=d_out)))
    _, g_ref = util.trimul_oracle(x, mask, w, "outgoing", d_out)
    cos_min, fro = util.TRIMUL_TOL[dtype, precision]
    for name, grad in grads.items():
        util.check_close("grad_" + name, grad, g_ref[name], cos_min, 2 * fro)   # (small sums: twice the tables' bound)


def test_unasked_sums_are_not_formed(tmu):
    """Without gradients of the input weights the input gate's backward has no products over the pixels."""
    from geometric_nn_ops_b200 import _lib
    x, mask, w, d_out = util.trimul_inputs(1, 64, 128, 128, torch.bfloat16)
    flops = {}
    for frozen in (False, True):
        leaves = [v.requires_grad_(not (frozen and k in ("p_in_weight", "g_in_weight"))) for k, v in {"x": x, **w}.items()]
        out = tmu(x, "outgoing", mask, **w)
        _lib.profile_enable(True)
        torch.autograd.grad(out, [v for v in leaves if v.requires_grad], grad_outputs=d_out)
        torch.cuda.synchronize()
        flops[frozen] = _lib.profile_summary()["tc_gate_in_bwd"][2]
        _lib.profile_enable(False)
    assert flops[False] > 0 and flops[True] == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=str)
@pytest.mark.parametrize("n", [8, 64, 72, 200])
def test_layernorm_sums_keep_their_order(n, dtype):
    """The means of both LayerNorms, bit for bit: a row's even and odd pairs of channels as two chains of additions; parts of 16 channels of
    the contraction.  Another order flips last bits of z and u, which a stack in 16 bits carries on."""
    import ctypes
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle._trimul import _DTYPES
    lib, M = _lib.load(), n * n
    x, mask, w, _ = util.trimul_inputs(1, n, 128, 128, dtype, seed=n)
    d = _lib.TriMulDesc(1, n, 128, 128, _DTYPES[dtype], _lib.PREC_IEEE, _lib.OUTGOING, 1e-5)
    wp = _lib.TriMulWeights(**{_lib.abi_field(k): t.data_ptr() for k, t in w.items()})
    saved = torch.empty(lib.tri_mul_saved_bytes(ctypes.byref(d)), dtype=torch.uint8, device="cuda")
    ws = torch.empty(lib.tri_mul_ws_bytes(ctypes.byref(d), 0), dtype=torch.uint8, device="cuda")
    out, at = torch.empty_like(x), lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.check(lib.tri_mul_fwd(ctypes.byref(d), at(x), at(mask), ctypes.byref(wp), at(out), at(saved), at(ws), ws.numel(),
                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "fwd")
    saved = saved.cpu()
    unit, room = -(-M * 256 // 256) * 256, -(-M * 4 // 256) * 256   # z, a, b, t, u; then mean, rstd of either LayerNorm
    floats = lambda i: saved[5 * unit + i * room:][:M * 4].view(torch.float32)  # noqa: E731
    rows = x.reshape(M, 64, 2).cpu().float()
    k = rows[:, 0, 0]
    chain = [torch.zeros(M, 2), torch.zeros(M, 2)]
    for i in range(64):
        chain[i & 1] = chain[i & 1] + (rows[:, i] - k[:, None])
    s = [c[:, 0] + c[:, 1] for c in chain]
    assert torch.equal(floats(0), (s[0] + s[1]) / 128 + k)
    t = saved[3 * unit:][:M * 256].view(dtype).reshape(8, 16, M).float()
    mean = torch.zeros(M)
    for part in t:
        s = torch.zeros(M)
        for c in part:
            s = s + (c - part[0])
        mean = mean + (s / 16 + part[0])
    assert torch.equal(floats(2), mean / 8)
