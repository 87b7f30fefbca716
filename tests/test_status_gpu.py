"""The status of kernels that start a call by themselves: every CTA reports in a byte of its own, whatever the workspace held before.

A CTA that starts late can then not take back what another has reported.  No wait is made to run out: the code is written in its place.
"""

import ctypes

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu


def _p(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def _reports(ws, ctas):
    """Nothing reported; then the code of any CTA is read back."""
    from geometric_nn_ops_b200 import _lib
    lib, stream = _lib.load(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.tri_ws_status(_p(ws), stream) == 0
    assert ws[:8].view(torch.int32).tolist() == [0, ctas]
    for cta in (0, 1, ctas // 2, ctas - 1):
        ws[8 + cta] = 77
        assert lib.tri_ws_status(_p(ws), stream) == -4 and b"code 77" in lib.tri_last_error(), cta
        ws[8 + cta] = 0
    assert lib.tri_ws_status(_p(ws), stream) == 0


# heads of up to 32 channels; of 64, one CTA per SM and more CTAs than SMs; TF32
@pytest.mark.parametrize("S,n,H,dim,dtype,ctas", [(20, 320, 2, 32, torch.bfloat16, 120), (60, 257, 2, 64, torch.float16, 296), (5, 64, 1, 64, torch.bfloat16, 5),
                                                  (80, 256, 4, 32, torch.float32, 148)], ids=lambda v: str(v).replace("torch.", ""))
def test_attention_forward(S, n, H, dim, dtype, ctas):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import _triattn, triangle_attention
    t, mask, _ = util.attn_inputs(1, S, n, H, dim, dtype, seed=n)
    precision = "tf32" if dtype == torch.float32 else "ieee"
    with torch.no_grad(), util.matmul_precision(precision):
        want = triangle_attention(t["q"], t["k"], t["v"], t["bias"], mask)
    m = mask.reshape(1, S, n).contiguous().view(torch.uint8)
    o, lse = torch.empty_like(t["q"]), torch.empty(2, 1, S, H, n, device="cuda")
    d = _triattn._desc(t["q"], t["k"], t["v"], o, t["bias"], m, dim ** -0.5, precision)
    size = _lib.load().tri_attn_ws_bytes(ctypes.byref(d), 0)
    ws = torch.full((size + 256,), 0x5A, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.load().tri_attn_fwd(ctypes.byref(d), _p(t["q"]), _p(t["k"]), _p(t["v"]), _p(t["bias"]), _p(m), _p(o), _p(lse), _p(ws), size,
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "fwd")
    assert _lib.last_path() == "tcgen05" and torch.equal(o, want) and bool((ws[size:] == 0x5A).all())
    _reports(ws, ctas)


@pytest.mark.parametrize("M,ctas", [(40 * 40, 13), (200 * 200, 148)])
def test_pair_bias_projection(M, ctas):
    """The first kernel of a call of attention_pair_bias, in the 256 bytes that it asks for."""
    from geometric_nn_ops_b200 import _lib
    g = torch.Generator().manual_seed(M)
    z, w = torch.randn(M, 128, generator=g).bfloat16().cuda(), torch.randn(8, 128, generator=g).bfloat16().cuda()
    bias = torch.empty(1, 8, M, dtype=torch.bfloat16, device="cuda")
    d = _lib.TriAttnProjDesc(M, 128, 8, 32, _lib.BF16, _lib.PREC_IEEE, 1e-5)
    ws = torch.full((512,), 0x5A, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.load().tri_attn_project_bias(ctypes.byref(d), M, _p(z), None, None, _p(w), _p(bias), _p(ws),
                                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "bias")
    want = torch.nn.functional.layer_norm(z.double(), (128,)).bfloat16().double() @ w.double().T
    assert float((bias[0].double().T - want).norm() / want.norm()) < 2.0 ** -8 and bool((ws[256:] == 0x5A).all())
    _reports(ws, ctas)
