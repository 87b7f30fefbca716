"""The multiplicative update at sides that are not a multiple of eight, on the tensor-core path, against the oracle."""

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

CASES = [(1, 1, False), (1, 9, True), (2, 31, False), (1, 129, False), (1, 203, True)]   # B, N, biases


@pytest.mark.parametrize("direction", ["outgoing", "incoming"])
@pytest.mark.parametrize("case", CASES, ids=str)
@pytest.mark.parametrize("dtype,precision", [(torch.bfloat16, "ieee"), (torch.float16, "ieee"), (torch.float32, "tf32")],
                         ids=lambda v: str(v).replace("torch.", ""))
def test_against_oracle(case, dtype, precision, direction):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import trimul_b200
    B, N, biases = case
    x, mask, w, d_out = util.trimul_inputs(B, N, 128, 128, dtype, seed=N, biases=biases, with_mask=N != 31)
    if N <= 9:
        d_out = torch.ones_like(d_out)     # a handful of pixels: a random d_out cancels in some of the weight gradients
    with util.matmul_precision(precision):
        out, grads = util.trimul_fwd_bwd(trimul_b200, x, mask, w, direction, d_out)
    torch.cuda.synchronize()
    assert _lib.last_path() == "tcgen05"
    o_ref, g_ref = util.trimul_oracle(x, mask, w, direction, d_out)
    cos_min, fro = util.TRIMUL_TOL[dtype, precision]
    util.check_close("out", out, o_ref, cos_min, fro)
    for name, val in grads.items():
        if N > 9:
            util.check_close("grad_" + name, val, g_ref[name], cos_min, fro)
        else:
            assert torch.isfinite(val.float()).all(), name


@pytest.mark.parametrize("B,N", [(1, 31), (2, 13), (1, 130)], ids=str)
@pytest.mark.parametrize("dtype,precision", [(torch.bfloat16, "ieee"), (torch.float32, "tf32")], ids=lambda v: str(v).replace("torch.", ""))
def test_eps_zero(B, N, dtype, precision):
    """Without an epsilon the pads' variance of zero must stay with the pads."""
    import functools

    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import trimul_b200
    from oracle import triangle_oracle as orc
    x, mask, w, d_out = util.trimul_inputs(B, N, 128, 128, dtype, seed=N)
    with util.matmul_precision(precision):
        out, grads = util.trimul_fwd_bwd(functools.partial(trimul_b200, eps=0.0), x, mask, w, "outgoing", d_out)
    torch.cuda.synchronize()
    assert _lib.last_path() == "tcgen05"
    wn = {k: util.f64(v) for k, v in w.items()}
    args = (util.f64(x), "outgoing", util.f64(mask))
    cos_min, fro = util.TRIMUL_TOL[dtype, precision]
    util.check_close("out", out, orc.trimul_fwd(*args, eps=0.0, **wn), cos_min, fro)
    g_ref = orc.trimul_bwd(*args, util.f64(d_out), eps=0.0, **wn)
    for name, val in grads.items():
        util.check_close("grad_" + name, val, g_ref[name], cos_min, fro)
