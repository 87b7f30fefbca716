"""Workspaces hold what a call needs: no copy of a bias that is read in place, one of a bias that all batch entries share."""

import ctypes

import pytest
import torch

from tests import util


def _attn_bytes(B, S, N, H, D, bias_st, is_bwd=0):
    from geometric_nn_ops_b200 import _lib
    d = _lib.TriAttnDesc()
    d.B, d.n_seq, d.n_res, d.H, d.D, d.dtype, d.scale = B, S, N, H, D, _lib.BF16, 1.0
    d.bias_st = (ctypes.c_int64 * 3)(*bias_st)
    return _lib.load().tri_attn_ws_bytes(ctypes.byref(d), is_bwd)


@pytest.mark.parametrize("is_bwd", [0, 1])
def test_attention_bias_copies(is_bwd):
    in_place = _attn_bytes(4, 64, 256, 4, 32, (4 * 256 * 256, 256 * 256, 256), is_bwd)
    shared = _attn_bytes(4, 64, 256, 4, 32, (0, 256 * 256, 256), is_bwd)
    broadcast = _attn_bytes(4, 64, 256, 4, 32, (0, 0, 0), is_bwd)
    plane = 4 * 256 * 256 * 2
    assert broadcast - shared == plane                        # heads and queries without a stride: one padded copy
    assert in_place - shared == (3 * plane if is_bwd else 0)  # the backward's transposed copies
    if not is_bwd:
        assert shared < 4 * 64 * 256 * 4 + 4096               # the mask terms and little else


def _tf32_desc(S, N, H, bias_st):
    from geometric_nn_ops_b200 import _lib
    d = _lib.TriAttnDesc()
    d.B, d.n_seq, d.n_res, d.H, d.D, d.dtype, d.precision, d.scale = 1, S, N, H, 32, _lib.F32, _lib.PREC_TF32, 1.0
    st = (ctypes.c_int64 * 4)(S * N * H * 32, N * H * 32, H * 32, 32)
    d.q_st = d.k_st = d.v_st = d.o_st = d.do_st = d.dq_st = d.dk_st = d.dv_st = st
    d.bias_st = (ctypes.c_int64 * 3)(*bias_st)
    return d


@pytest.mark.parametrize("is_bwd", [0, 1])
def test_tf32_attention(is_bwd):
    from geometric_nn_ops_b200 import _lib
    size = lambda *a: _lib.load().tri_attn_ws_bytes(ctypes.byref(_tf32_desc(*a)), is_bwd)  # noqa: E731
    S, N, H = 96, 256, 4
    plane, tensor = H * N * N * 4, S * N * H * 32 * 4
    in_place, broadcast = size(S, N, H, (0, N * N, N)), size(S, N, H, (0, 0, N))
    assert broadcast - in_place == plane                 # one bias for all heads: a copy per head
    if not is_bwd:
        assert in_place < 3 * tensor + S * N * 4 + 4096  # q, k, v rounded, the mask terms


@pytest.mark.parametrize("N,chunks", [(768, 1), (256, 8)])
def test_attention_bias_gradient_partials(N, chunks):
    """A partial sum per row chunk, none where one CTA has all rows of a tile (148 SMs, two CTAs each)."""
    S, H, D = N, 4, 32
    blocks, rows = (N + 127) // 128, S * H
    npad = blocks * 128
    rest = 512 + blocks * rows * N * D * 2 + rows * npad * (3 * 4 + 16) + 2 * S * npad * 4 + rows * 4 + H * N * N * 2
    partials = (chunks if chunks > 1 else 0) * H * N * N * 4
    assert 0 <= _attn_bytes(1, S, N, H, D, (0, N * N, N), 1) - rest - partials < 8 * 256


def test_ragged_update_forward():
    from geometric_nn_ops_b200 import _lib
    size = lambda n: _lib.load().tri_mul_ws_bytes(ctypes.byref(_lib.TriMulDesc(1, n, 128, 128, _lib.BF16, 0, 0, 1e-5)), 0)  # noqa: E731
    assert size(203) - size(208) <= 208 * 208 * 2 + 1024      # a padded mask, no padded x and out


def test_update_backward():
    from geometric_nn_ops_b200 import _lib
    lib = _lib.load()
    size = lambda b: lib.tri_mul_ws_bytes(ctypes.byref(_lib.TriMulDesc(b, 256, 128, 128, _lib.BF16, 0, 0, 1e-5)), 1)  # noqa: E731
    unit = 256 * 256 * 128 * 2
    # per pixel and channel: dy, dgo, dt, da, db, four of dPG; du for batches only, where the LayerNorm's backward reads it
    fixed = size(1) - 9 * unit
    assert 0 < fixed < 48 << 20 and size(2) == fixed + 2 * 10 * unit
    phase = lambda b: lib.tri_mul_shard_ws_bytes(ctypes.byref(_lib.TriMulShardDesc(b, 256, 256, 128, 128, _lib.BF16, 0, 1e-5)), _lib.PHASE_OUTPUT_BWD)  # noqa: E731
    assert phase(2) - phase(1) == 3 * unit


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.gpu
@pytest.mark.parametrize("room", [True, False])
def test_attention_bias_off_16_bytes(room):
    """A bias that starts off a 16-byte boundary: copied where the workspace has room, else read by the CUDA-core kernels."""
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import _triattn, triangle_attention
    t, mask, d_out = util.attn_inputs(1, 4, 136, 2, 32, torch.bfloat16, seed=3)
    want, g_want = util.attn_fwd_bwd(triangle_attention, t, mask, None, d_out)
    flat = torch.empty(t["bias"].numel() + 1, dtype=torch.bfloat16, device="cuda")
    bias = flat[1:].view(t["bias"].shape).copy_(t["bias"])
    if room:
        leaves = {n: t[n].clone().requires_grad_() for n in ("q", "k", "v")}
        flat.requires_grad_()
        view = flat[1:].view(t["bias"].shape)
        out = triangle_attention(leaves["q"], leaves["k"], leaves["v"], view, mask)
        got = torch.autograd.grad(out, [*leaves.values(), view], grad_outputs=d_out)
        torch.cuda.synchronize()
        assert _lib.last_path() == "tcgen05" and torch.equal(out, want)
        for name, g in zip(("q", "k", "v", "bias"), got):
            assert torch.equal(g, g_want[name]), name
        return
    lib, q = _lib.load(), t["q"]
    m = mask.reshape(1, 4, 136).contiguous().view(torch.uint8)
    o, lse = torch.empty_like(q), torch.empty(2, 1, 4, 2, 136, device="cuda")
    d = _triattn._desc(q, t["k"], t["v"], o, bias, m, 32 ** -0.5, "ieee")
    ws = torch.empty(lib.tri_attn_ws_bytes(ctypes.byref(d), 0), dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(lib.tri_attn_fwd(ctypes.byref(d), _p(q), _p(t["k"]), _p(t["v"]), _p(bias), _p(m), _p(o), _p(lse), _p(ws), ws.numel(), stream), "fwd")
    torch.cuda.synchronize()
    assert _lib.last_path() == "simt"
    util.check_close("out", o, util.f64(want), *util.ATTN_TOL[torch.bfloat16, "ieee"])


@pytest.mark.gpu
def test_tf32_bias_off_16_bytes():
    """The same for fp32 with TF32 products: a copy where there is room, else the CUDA-core kernels."""
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import triangle_attention
    S, N, H = 96, 256, 4
    t, mask, d_out = util.attn_inputs(1, S, N, H, 32, torch.float32, seed=3)
    flat = torch.empty(t["bias"].numel() + 1, device="cuda", requires_grad=True)
    with torch.no_grad():
        flat[1:].copy_(t["bias"].flatten())
    with util.matmul_precision("tf32"):
        want, g_want = util.attn_fwd_bwd(triangle_attention, t, mask, None, d_out)
        leaves = {n: t[n].clone().requires_grad_() for n in ("q", "k", "v")}
        view = flat[1:].view(t["bias"].shape)
        out = triangle_attention(leaves["q"], leaves["k"], leaves["v"], view, mask)
        got = torch.autograd.grad(out, [*leaves.values(), view], grad_outputs=d_out)
    torch.cuda.synchronize()
    assert _lib.last_path() == "tcgen05" and torch.equal(out, want)
    for name, g in zip(("q", "k", "v", "bias"), got):
        assert torch.equal(g, g_want[name]), name
    lib, q = _lib.load(), t["q"]
    m = mask.reshape(1, S, N).contiguous().view(torch.uint8)
    o, lse = torch.empty_like(q), torch.empty(2, 1, S, H, N, device="cuda")
    d = _tf32_desc(S, N, H, (0, N * N, N))
    d.scale, d.mask_st = 32 ** -0.5, (ctypes.c_int64 * 2)(S * N, N)
    n = lib.tri_attn_ws_bytes(ctypes.byref(d), 0)
    for extra, path in ((0, "simt"), (4 * H * N * (N + 7) + 256, "tcgen05")):
        ws = torch.empty(n + extra, dtype=torch.uint8, device="cuda")
        _lib.check(lib.tri_attn_fwd(ctypes.byref(d), _p(q), _p(t["k"]), _p(t["v"]), _p(view.detach()), _p(m), _p(o), _p(lse), _p(ws), ws.numel(),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "fwd")
        torch.cuda.synchronize()
        assert _lib.last_path() == path
        util.check_close("out", o, util.f64(want.detach()), *util.ATTN_TOL[torch.float32, "tf32"])
