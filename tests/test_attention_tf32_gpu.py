"""fp32 triangle attention with TF32 products on the tensor cores, against softmax over fp32 logits with fp64 products.

Every operand of a product is rounded to eleven bits: a relative error of up to 2^-12 in q, k, v, P, dO and dS each.  The logits'
error enters P (and dS) about once more; 4 * 2^-12 bounds the 2-norm of all six together.
"""

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu
LIMIT = 4 * 2.0 ** -12


def _reference(t, mask, d_out, scale):
    heads = lambda x: x.transpose(2, 3).double()  # noqa: E731
    q, k, v, do = (heads(x) for x in (t["q"], t["k"], t["v"], d_out))
    x = (q @ k.transpose(-1, -2) * scale).float()
    if t["bias"] is not None:
        x = x + t["bias"]
    if mask is not None:
        x = x + 1e9 * (mask.float() - 1)
    p = torch.softmax(x.double(), -1)
    dp = do @ v.transpose(-1, -2)
    ds = p * (dp - (dp * p).sum(-1, keepdim=True))
    back = lambda x: x.transpose(2, 3)  # noqa: E731
    grads = {"q": back(ds @ k) * scale, "k": back(ds.transpose(-1, -2) @ q) * scale, "v": back(p.transpose(-1, -2) @ do),
             "bias": ds.sum(1, keepdim=True)}
    return back(p @ v), grads


def _check(t, mask, d_out, path="tcgen05"):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import triangle_attention
    with util.matmul_precision("tf32"):
        out, grads = util.attn_fwd_bwd(triangle_attention, t, mask, None, d_out)
    torch.cuda.synchronize()
    assert _lib.last_path() == path
    o_ref, g_ref = _reference(t, mask, d_out, t["q"].shape[-1] ** -0.5)
    for name, got in (("out", out.detach()), *grads.items()):
        want = o_ref if name == "out" else g_ref[name]
        assert torch.isfinite(got).all(), name
        err = float((got.double() - want).norm() / want.norm())
        assert err <= LIMIT, f"{name}: {err:.2e} > {LIMIT:.2e}"


# the smallest calls of either direction, one and a half blocks, odd numbers of tiles, of rows and of columns, narrow heads
@pytest.mark.parametrize("shape", [(1, 80, 256, 4, 32), (1, 40, 256, 2, 32), (2, 62, 301, 2, 32), (1, 511, 140, 2, 32), (1, 103, 320, 2, 16),
                                   (1, 401, 129, 3, 32), (1, 240, 170, 3, 20), (1, 2, 1800, 4, 8), (1, 2000, 72, 2, 32)], ids=str)
def test_forward_and_backward(shape):
    t, mask, d_out = util.attn_inputs(*shape, torch.float32, seed=sum(shape), keep=0.9)
    t["q"] *= 0.5             # logits of q and k within 16: beside -1e9 they are lost, in whatever order
    mask[0, 1] = False        # a row with no key at all
    _check(t, mask, d_out)


@pytest.mark.parametrize("level", [300.0, -1e9, float("-inf"), 1e8])
def test_rows_without_factors(level):
    t, mask, d_out = util.attn_inputs(1, 70, 288, 4, 32, torch.float32, seed=5, keep=0.95)
    t["q"] *= 0.5
    t["bias"][..., 7, :64] = level
    t["bias"][..., 40, :-1] = level
    t["bias"][..., 70:75, ::2] = level
    mask[0, 0, ..., -1] = True
    mask[..., 3] = True
    _check(t, mask, d_out)


@pytest.mark.parametrize("kind", ["no bias", "no mask", "bias of one head", "transposed tokens", "batch of two"])
def test_operands(kind):
    B = 2 if kind == "batch of two" else 1
    t, mask, d_out = util.attn_inputs(B, 160 // B, 260, 2, 32, torch.float32, seed=9, keep=0.9, with_bias=kind != "no bias", with_mask=kind != "no mask")
    if kind == "bias of one head":
        t["bias"] = t["bias"][:, :, :1].expand(-1, -1, 2, -1, -1)
    if kind == "transposed tokens":
        for name in "qkv":
            t[name] = t[name].transpose(2, 3).contiguous().transpose(2, 3)
    if kind == "bias of one head":   # (its gradient is that of the expanded view)
        from geometric_nn_ops_b200.triangle import triangle_attention
        leaf = t["bias"].detach()
        with util.matmul_precision("tf32"):
            out = triangle_attention(t["q"], t["k"], t["v"], leaf, mask)
        o_ref, _ = _reference({**t, "bias": leaf}, mask, d_out, 32 ** -0.5)
        assert float((out.double() - o_ref).norm() / o_ref.norm()) <= LIMIT
        return
    _check(t, mask, d_out)


def test_scratch_limit():
    """A workspace below what the tensor cores ask for is served by the CUDA-core path, as before."""
    import ctypes

    from geometric_nn_ops_b200 import _lib
    d = _lib.TriAttnDesc()
    d.B, d.n_seq, d.n_res, d.H, d.D, d.dtype, d.precision, d.scale = 1, 80, 256, 4, 32, _lib.F32, _lib.PREC_TF32, 1.0
    full = _lib.load().tri_attn_ws_bytes(ctypes.byref(d), 0)
    assert full >= 3 * 80 * 256 * 4 * 32 * 4
    st = (ctypes.c_int64 * 4)(80 * 256 * 128, 256 * 128, 128, 32)
    d.q_st = d.k_st = d.v_st = d.o_st = st
    d.bias_st = (ctypes.c_int64 * 3)(0, 8, 8)
    q, k, v = (torch.randn(1, 80, 256, 4, 32, device="cuda") for _ in range(3))
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    outs = []
    for n in (full, 4096):
        o, stats, ws = torch.empty_like(q), torch.empty(2, 1, 80, 4, 256, device="cuda"), torch.empty(n, dtype=torch.uint8, device="cuda")
        _lib.check(_lib.load().tri_attn_fwd(ctypes.byref(d), p(q), p(k), p(v), None, None, p(o), p(stats), p(ws), ctypes.c_size_t(n),
                                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "tri_attn_fwd")
        torch.cuda.synchronize()
        outs.append((o, _lib.last_path()))
    assert [x[1] for x in outs] == ["tcgen05", "simt"]
    assert float((outs[0][0] - outs[1][0]).norm() / outs[1][0].norm()) <= LIMIT
