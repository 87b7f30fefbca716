"""The one-kernel LayerNorm + projection (16-bit types, 128 channels) against fp32 torch on the rounded inputs, where its
tiling can go wrong: fewer pixels than a tile, a ragged last tile, more tiles than SMs, two batch entries that share a
tile, head counts up to the limit, output widths that are not whole blocks."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _operands(B, U, V, H, n_out, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    z = torch.randn(B, U, V, 128, generator=g) * 2 + 3 * torch.randn(B, U, V, 1, generator=g)
    w = [torch.randn(n, 128, generator=g) * 128 ** -0.5 for n in (H, max(n_out, 1))]
    ln = 1 + 0.1 * torch.randn(128, generator=g)
    return [t.to(dtype).cuda() for t in (z, ln, *w)]


def _close(got, want, dtype):
    rel = (got.float() - want).norm() / want.norm()
    assert rel < (6e-3 if dtype == torch.bfloat16 else 1e-3), rel


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=str)
@pytest.mark.parametrize("B,U,V,H", [(1, 1, 1, 1), (2, 5, 7, 16), (1, 129, 1, 5), (3, 90, 77, 8), (1, 200, 190, 16)])
def test_pair_bias(B, U, V, H, dtype):
    from geometric_nn_ops_b200 import _lib
    z, ln, w, _ = _operands(B, U, V, H, 0, dtype, U + V)
    for weight in (ln, None):
        with torch.no_grad():
            got = _lib.host().pair_bias(z, weight, w, 1e-5)
        zn = F.layer_norm(z.float(), (128,), None if weight is None else weight.float(), None, 1e-5).to(dtype).float()
        assert got.is_contiguous() and got.shape == (B, H, U, V)
        _close(got, (zn @ w.float().t()).permute(0, 3, 1, 2), dtype)


@pytest.mark.parametrize("H,D,pixels", [(1, 8, 127), (5, 8, 128), (4, 24, 129), (8, 16, 20000)])
def test_projection(H, D, pixels):
    from geometric_nn_ops_b200.triangle import attention_input_projection
    dtype = torch.bfloat16
    z, ln, wb, wq = _operands(1, 1, pixels, H, 3 * H * D, dtype, pixels)
    with torch.no_grad():
        q, k, v, bias = attention_input_projection(z, wq, wb, H, ln)
    zn = F.layer_norm(z.float(), (128,), ln.float()).to(dtype).float()
    ref = (zn @ wq.float().t()).view(1, 1, pixels, 3, H, D)
    for got, want in ((q, ref[..., 0, :, :]), (k, ref[..., 1, :, :]), (v, ref[..., 2, :, :]), (bias, (zn @ wb.float().t()).permute(0, 3, 1, 2))):
        _close(got, want, dtype)


def test_pair_bias_leaves_other_calls_to_torch():
    from geometric_nn_ops_b200 import _lib
    z, ln, w, _ = _operands(1, 4, 4, 4, 0, torch.bfloat16, 0)
    fits = _lib.host().pair_bias_fits
    assert fits(z, ln, w) and fits(z, None, w)
    assert not fits(z.float(), ln.float(), w.float()) and not fits(z, ln, w.requires_grad_())
    assert not fits(z[..., :64].contiguous(), ln[:64], w.detach()[:, :64])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16], ids=str)
@pytest.mark.parametrize("n,offset", [(1, 0), (7, 0), (2048, 0), (5000, 0), (4096, 1)])
def test_gate_mul(n, offset, dtype):
    import ctypes

    from geometric_nn_ops_b200 import _lib
    g = torch.Generator().manual_seed(n)
    a, gate = ((torch.randn(n + offset, generator=g) * 3).to(dtype).cuda()[offset:] for _ in range(2))
    out = torch.full((n + 8,), 7.0, dtype=dtype, device="cuda")
    code = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16, torch.float16: _lib.F16}[dtype]
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _lib.check(_lib.load().tri_gate_mul(code, n, p(a), p(gate), p(out), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "tri_gate_mul")
    want = (a.float() * torch.sigmoid(gate.float())).to(dtype)
    assert torch.allclose(out[:n].float(), want.float(), rtol=1e-6 if dtype == torch.float32 else 8e-3, atol=1e-6) and (out[n:] == 7).all()
