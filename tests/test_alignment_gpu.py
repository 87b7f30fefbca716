"""Tensors that start off the boundaries the kernels' wide accesses like: views into a flat buffer, and pointers through the C ABI."""

import ctypes

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu


def _at(t, elements):
    """A copy of t that starts `elements` into its storage."""
    flat = torch.empty(t.numel() + 64, dtype=t.dtype, device=t.device)
    out = flat[elements:elements + t.numel()].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=str)
@pytest.mark.parametrize("B,n", [(1, 40), (2, 24)])
def test_update_gradient_on_16_but_not_32_bytes(B, n, dtype):
    from geometric_nn_ops_b200.triangle import trimul_b200
    x, mask, w, d_out = util.trimul_inputs(B, n, 128, 128, dtype, seed=n)
    out, want = util.trimul_fwd_bwd(trimul_b200, x, mask, w, "outgoing", d_out)
    out8, got = util.trimul_fwd_bwd(trimul_b200, _at(x, 8), mask, w, "outgoing", _at(d_out, 8))
    assert _at(d_out, 8).data_ptr() % 32 == 16 and torch.equal(out8, out)
    for name in want:
        assert torch.equal(got[name], want[name]), name


def _p(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def test_attention_results_off_16_bytes():
    """Results that cannot be written in 16-byte pieces come from the CUDA-core kernels."""
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import _triattn
    lib = _lib.load()
    t, mask, d_o = util.attn_inputs(1, 4, 64, 2, 32, torch.bfloat16, seed=1)
    q, k, v, bias = t["q"], t["k"], t["v"], t["bias"]
    m = mask.reshape(1, 4, 64).contiguous().view(torch.uint8)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def call(off):
        new = lambda like, n: _at(torch.zeros_like(like), n)  # noqa: E731
        o, (dq, dk, dv) = new(q, off), (new(q, off) for _ in range(3))
        dbias = _at(torch.zeros(1, 2, 64, 64, device="cuda"), off)
        lse = torch.empty(2, 1, 4, 2, 64, device="cuda")
        d = _triattn._desc(q, k, v, o, bias, m, 32 ** -0.5, "ieee")
        d.do_st = d.dq_st = d.dk_st = d.dv_st = _triattn._st4(q)
        ws = torch.empty(max(lib.tri_attn_ws_bytes(ctypes.byref(d), b) for b in (0, 1)), dtype=torch.uint8, device="cuda")
        _lib.check(lib.tri_attn_fwd(ctypes.byref(d), _p(q), _p(k), _p(v), _p(bias), _p(m), _p(o), _p(lse), _p(ws), ws.numel(), stream), "fwd")
        path = [_lib.last_path()]
        _lib.check(lib.tri_attn_bwd(ctypes.byref(d), _p(q), _p(k), _p(v), _p(bias), _p(m), _p(o), _p(lse), _p(d_o), _p(dq), _p(dk), _p(dv),
                                    _p(dbias), _p(ws), ws.numel(), stream), "bwd")
        torch.cuda.synchronize()
        return path + [_lib.last_path()], {"o": o, "dq": dq, "dk": dk, "dv": dv, "dbias": dbias}

    path, want = call(0)
    assert path == ["tcgen05", "tcgen05"]
    path, got = call(1)
    assert path == ["simt", "simt"]
    cos_min, fro = util.ATTN_TOL[torch.bfloat16, "ieee"]
    for name in want:
        util.check_close(name, got[name], util.f64(want[name]), cos_min, fro)


def test_update_refuses_results_off_16_bytes():
    from geometric_nn_ops_b200 import _lib
    lib = _lib.load()
    x, mask, w, _ = util.trimul_inputs(1, 16, 128, 128, torch.bfloat16, seed=1)
    d = _lib.TriMulDesc(1, 16, 128, 128, _lib.BF16, _lib.PREC_IEEE, _lib.OUTGOING, 1e-5)
    wp = _lib.TriMulWeights(**{_lib.abi_field(n): (t.data_ptr() if t is not None else None) for n, t in ((n, w.get(n)) for n in _lib.WEIGHT_NAMES)})
    ws = torch.empty(lib.tri_mul_ws_bytes(ctypes.byref(d), 0), dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    call = lambda out: lib.tri_mul_fwd(ctypes.byref(d), _p(x), _p(mask), ctypes.byref(wp), _p(out), None, _p(ws), ws.numel(), stream)  # noqa: E731
    assert call(_at(torch.empty_like(x), 4)) == -1 and b"16-byte" in lib.tri_last_error()
    assert call(_at(torch.empty_like(x), 8)) == 0
    torch.cuda.synchronize()


@pytest.mark.parametrize("dtype,precision,S,N,offset,paths", [
    (torch.bfloat16, "ieee", 4, 136, 0, ["tcgen05", "tcgen05"]), (torch.bfloat16, "ieee", 4, 136, 16, ["tcgen05", "simt"]),
    (torch.bfloat16, "ieee", 4, 136, 8, ["simt", "simt"]), (torch.bfloat16, "ieee", 4, 136, 4, ["simt", "simt"]),
    (torch.float32, "tf32", 80, 256, 16, ["tcgen05", "tcgen05"]), (torch.float32, "tf32", 80, 256, 4, ["simt", "simt"])],
    ids=lambda v: str(v).replace("torch.", "") if not isinstance(v, list) else "-".join(v))
def test_attention_workspace_off_its_boundary(dtype, precision, S, N, offset, paths):
    """A workspace that the tensor-core kernels cannot use is served by the CUDA-core kernels."""
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import _triattn, triangle_attention
    lib, H = _lib.load(), 4
    t, mask, d_o = util.attn_inputs(1, S, N, H, 32, dtype, seed=2)
    with util.matmul_precision(precision):
        want, g_want = util.attn_fwd_bwd(triangle_attention, t, mask, None, d_o)
    q, k, v, bias = t["q"], t["k"], t["v"], t["bias"]
    m = mask.reshape(1, S, N).contiguous().view(torch.uint8)
    o, dq, dk, dv = (torch.empty_like(q) for _ in range(4))
    dbias, lse = torch.empty(1, H, N, N, device="cuda"), torch.empty(2, 1, S, H, N, device="cuda")
    d = _triattn._desc(q, k, v, o, bias, m, 32 ** -0.5, precision)
    d.do_st = d.dq_st = d.dk_st = d.dv_st = _triattn._st4(q)
    n = max(lib.tri_attn_ws_bytes(ctypes.byref(d), b) for b in (0, 1))
    ws = torch.empty(n + 64, dtype=torch.uint8, device="cuda")
    assert ws.data_ptr() % 32 == 0
    at, stream = ctypes.c_void_p(ws.data_ptr() + offset), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(lib.tri_attn_fwd(ctypes.byref(d), _p(q), _p(k), _p(v), _p(bias), _p(m), _p(o), _p(lse), at, n, stream), "fwd")
    path = [_lib.last_path()]
    _lib.check(lib.tri_attn_bwd(ctypes.byref(d), _p(q), _p(k), _p(v), _p(bias), _p(m), _p(o), _p(lse), _p(d_o), _p(dq), _p(dk), _p(dv),
                                _p(dbias), at, n, stream), "bwd")
    torch.cuda.synchronize()
    assert path + [_lib.last_path()] == paths
    cos_min, fro = util.ATTN_TOL[dtype, precision]
    for name, got, ref in (("out", o, want.detach()), ("dq", dq, g_want["q"]), ("dk", dk, g_want["k"]), ("dv", dv, g_want["v"]),
                           ("dbias", dbias, g_want["bias"].reshape(dbias.shape))):
        util.check_close(name, got, util.f64(ref), cos_min, fro)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=str)
@pytest.mark.parametrize("B,n", [(1, 64), (2, 32), (1, 43)])
def test_update_scratch_on_16_but_not_32_bytes(B, n, dtype):
    """ws and the saved block hold the gradients that the gate epilogues read and write in wide pieces."""
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle._trimul import _DTYPES
    lib = _lib.load()
    x, mask, w, d_out = util.trimul_inputs(B, n, 128, 128, dtype, seed=n)
    d = _lib.TriMulDesc(B, n, 128, 128, _DTYPES[dtype], _lib.PREC_TF32 if dtype == torch.float32 else _lib.PREC_IEEE, _lib.OUTGOING, 1e-5)
    wp = _lib.TriMulWeights(**{_lib.abi_field(k): t.data_ptr() for k, t in w.items()})
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    sizes = [lib.tri_mul_saved_bytes(ctypes.byref(d)), lib.tri_mul_ws_bytes(ctypes.byref(d), 0), lib.tri_mul_ws_bytes(ctypes.byref(d), 1)]

    def call(offset):
        saved, ws, ws_bwd = (torch.zeros(s + 64, dtype=torch.uint8, device="cuda") for s in sizes)
        at = [ctypes.c_void_p(t.data_ptr() + offset) for t in (saved, ws, ws_bwd)]
        out, dx = torch.empty_like(x), torch.empty_like(x)
        grads = {k: torch.empty(t.shape, device="cuda") for k, t in w.items()}
        g = _lib.TriMulWeightGrads(**{_lib.abi_field(k): t.data_ptr() for k, t in grads.items()})
        _lib.check(lib.tri_mul_fwd(ctypes.byref(d), _p(x), _p(mask), ctypes.byref(wp), _p(out), at[0], at[1], sizes[1], stream), "fwd")
        _lib.check(lib.tri_mul_bwd(ctypes.byref(d), _p(x), _p(mask), ctypes.byref(wp), at[0], _p(d_out), _p(dx), ctypes.byref(g), at[2], sizes[2],
                                   stream), "bwd")
        torch.cuda.synchronize()
        assert all(int(t[sizes[i] + offset:].sum()) == 0 and int(t[:offset].sum()) == 0 for i, t in enumerate((saved, ws, ws_bwd)))
        return {"out": out, "dx": dx, **grads}

    want, got = call(0), call(16)
    for name in want:
        assert torch.equal(got[name], want[name]), name


@pytest.mark.parametrize("dtype,H,D", [(torch.float32, 4, 32), (torch.float32, 3, 16), (torch.bfloat16, 4, 32), (torch.bfloat16, 8, 32)], ids=str)
def test_projection_of_views_off_16_bytes(dtype, H, D):
    """z and weights that are views into a flat buffer: copied by the Python entry, refused by the C entry before a launch."""
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import attention_input_projection
    g = torch.Generator().manual_seed(H)
    rn = lambda *s: torch.randn(*s, generator=g).to(dtype).cuda()  # noqa: E731
    args = [rn(1, 5, 40, 128), rn(3 * H * D, 128), rn(H, 128), rn(128), rn(128)]
    call = lambda z, wq, wb, lw, lb: attention_input_projection(z, wq, wb, H, lw, lb)  # noqa: E731
    with util.matmul_precision("tf32"), torch.no_grad():
        want = call(*args)
        for got, ref in zip(call(*(_at(t, 1) for t in args)), want):
            assert torch.equal(got, ref)
    if dtype == torch.bfloat16 and H == 4:
        return      # the one-kernel form: its norm weights are read one at a time
    z, wq, wb, lw, lb = args
    d = _lib.TriAttnProjDesc(200, 128, H, D, _lib.F32 if dtype == torch.float32 else _lib.BF16, _lib.PREC_TF32, 1e-5)
    n = _lib.load().tri_attn_project_ws_bytes(ctypes.byref(d))
    ws = torch.empty(n + 64, dtype=torch.uint8, device="cuda")
    qkv, bias = torch.empty(200, 3 * H * D, dtype=dtype, device="cuda"), torch.empty(H, 200, dtype=dtype, device="cuda")
    before = _lib.launch_count()
    for i in range(5):
        p = [_p(_at(t, 1) if j == i else t) for j, t in enumerate((z, lw, lb, wq))]
        at = ctypes.c_void_p(ws.data_ptr() + (4 if i == 4 else 0))
        assert _lib.load().tri_attn_project(ctypes.byref(d), *p, _p(wb), _p(qkv), _p(bias), at, n, None) == -1
    assert _lib.launch_count() == before
