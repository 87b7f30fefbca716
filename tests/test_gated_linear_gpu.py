"""tri_gated_linear, out = (o * sigmoid(s Wg^T)) Wo^T, at the edges of its tiles, against fp64.

The gated tensor is rounded to the operand type once and the result once more: 2^-9 and 2^-9 relative (bf16; 2^-12 fp16) per
element at most, so 2^-8 (2^-11) bounds the 2-norm.
"""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("M,K,W,N", [(1, 8, 8, 8), (3, 64, 40, 24), (127, 72, 128, 136), (128, 128, 136, 128), (129, 768, 264, 8), (385, 768, 768, 768),
                                     (2051, 136, 512, 200)])
def test_gated_linear(dtype, M, K, W, N):
    from geometric_nn_ops_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(M + K)
    rn = lambda *s, sc=1.0: (torch.randn(*s, generator=g, device="cuda") * sc).to(dtype)  # noqa: E731
    s, o, wg, wo = rn(M, K), rn(M, W), rn(W, K, sc=K ** -0.5), rn(N, W, sc=W ** -0.5)
    gated, out, status = torch.full_like(o, 7), torch.full((M + 1, N), 7, dtype=dtype, device="cuda"), torch.zeros(64, dtype=torch.int32, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    code = _lib.BF16 if dtype == torch.bfloat16 else _lib.F16
    _lib.check(_lib.load().tri_gated_linear(code, M, K, W, N, p(s), p(wg), p(o), p(wo), p(gated), p(out), p(status),
                                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "tri_gated_linear")
    torch.cuda.synchronize()
    assert int(status[0]) == 0 and (out[M:] == 7).all()      # nothing behind the last row
    ref_g = o.double() * torch.sigmoid(s.double() @ wg.double().t())
    ref = ref_g @ wo.double().t()
    limit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert float((gated.double() - ref_g).norm() / ref_g.norm()) <= limit
    assert float((out[:M].double() - ref).norm() / ref.norm()) <= limit


def _operands(M, W, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(M)
    rn = lambda *s, sc=1.0: (torch.randn(*s, generator=g, device="cuda") * sc).to(dtype)  # noqa: E731
    return rn(M, W), rn(M, W), rn(W, W, sc=W ** -0.5), rn(W, W, sc=3 * W ** -0.5)


def _call(f, M, W, s, wg, o, wo, gated, out, status):
    from geometric_nn_ops_b200 import _lib
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _lib.check(f(_lib.BF16, M, W, W, W, p(s), p(wg), p(o), p(wo), p(gated), p(out), p(status),
                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "tri_gated_linear")


@pytest.mark.parametrize("M,W", [(128, 256), (2048, 768), (9000, 256)])
def test_chained_calls(M, W):
    """s is what the call before wrote: nothing of it is read before that call is done."""
    from geometric_nn_ops_b200 import _lib
    f = _lib.load().tri_gated_linear
    s, o, wg, wo = _operands(M, W)
    status = torch.zeros(64, dtype=torch.int32, device="cuda")

    def chain(wait):
        bufs = [torch.full_like(s, float("nan")) for _ in range(8)]
        gated = [torch.empty_like(o) for _ in range(8)]
        torch.cuda.synchronize()
        x = s
        for out, scratch in zip(bufs, gated):
            _call(f, M, W, x, wg, o, wo, scratch, out, status)
            if wait:
                torch.cuda.synchronize()
            x = out
        torch.cuda.synchronize()
        return bufs

    want = chain(True)
    for _ in range(20):
        for got, ref in zip(chain(False), want):
            assert torch.equal(got, ref)
    assert int(status[0]) == 0


def test_behind_the_call_that_wrote_o():
    """The early form: o is what the call before wrote, s and the weights are older."""
    from geometric_nn_ops_b200 import _lib
    lib, M, W = _lib.load(), 2048, 768
    s, o, wg, wo = _operands(M, W)
    status = torch.zeros(64, dtype=torch.int32, device="cuda")
    mid, out, g1, g2 = (torch.full_like(s, float("nan")) for _ in range(4))
    want = torch.empty_like(out)
    _call(lib.tri_gated_linear, M, W, s, wg, o, wo, g1, mid, status)
    torch.cuda.synchronize()
    _call(lib.tri_gated_linear, M, W, s, wg, mid, wo, g2, want, status)
    torch.cuda.synchronize()
    for _ in range(20):
        mid.fill_(float("nan"))
        out.fill_(float("nan"))
        _call(lib.tri_gated_linear, M, W, s, wg, o, wo, g1, mid, status)
        _call(lib.tri_gated_linear_after, M, W, s, wg, mid, wo, g2, out, status)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert int(status[0]) == 0


def test_refusals():
    from geometric_nn_ops_b200 import _lib
    t = torch.zeros(64, dtype=torch.bfloat16, device="cuda")
    p = ctypes.c_void_p(t.data_ptr())
    off = ctypes.c_void_p(t.data_ptr() + 2)
    f = _lib.load().tri_gated_linear
    st = ctypes.c_void_p(0)
    assert f(_lib.F32, 1, 8, 8, 8, p, p, p, p, p, p, p, st) != 0
    assert f(_lib.BF16, 1, 12, 8, 8, p, p, p, p, p, p, p, st) != 0
    assert f(_lib.BF16, 1, 8, 8, 8, off, p, p, p, p, p, p, st) != 0
    assert f(_lib.BF16, 0, 8, 8, 8, p, p, p, p, p, p, p, st) != 0


@pytest.mark.parametrize("rows,n", [(1, 200), (1, 512), (1, 768), (1, 1000), (3, 200)])
def test_beside_an_attention(rows, n):
    """The gated product's tiles are as many as the attention before it leaves SMs, of 32, 64 or 128 columns: the result is the same."""
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import triangle_attention
    lib, H, D = _lib.load(), 16, 48
    M, W = rows * n, H * D
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v = (torch.randn(1, rows, n, H, D, generator=g, device="cuda").bfloat16() for _ in range(3))
    bias = torch.randn(1, 1, H, n, n, generator=g, device="cuda").bfloat16()
    s, _, wg, wo = _operands(M, W)
    status = torch.zeros(64, dtype=torch.int32, device="cuda")
    gated, out, g1, want = (torch.full_like(s, float("nan")) for _ in range(4))
    with torch.no_grad():
        o = triangle_attention(q, k, v, bias)
        torch.cuda.synchronize()
        _call(lib.tri_gated_linear, M, W, s, wg, o, wo, g1, want, status)
        torch.cuda.synchronize()
        for _ in range(5):
            out.fill_(float("nan"))
            torch.cuda.synchronize()
            o = triangle_attention(q, k, v, bias)
            assert _lib.last_path() == "tcgen05"
            _call(lib.tri_gated_linear_after, M, W, s, wg, o, wo, gated, out, status)
            torch.cuda.synchronize()
            assert torch.equal(gated, g1) and torch.equal(out, want)
    assert int(status[0]) == 0
