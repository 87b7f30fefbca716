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
