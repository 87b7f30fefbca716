"""Residual forms of the two ops: the same bits as the op followed by an addition."""

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=str)
@pytest.mark.parametrize("B,N", [(1, 8), (1, 24), (1, 200), (2, 16), (1, 21)])   # last two: the op, then an addition
def test_multiplicative_update(B, N, dtype):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import triangle_multiplicative_update as tmu
    x, mask, w, _ = util.trimul_inputs(B, N, 128, 128, dtype, seed=N, biases=True)
    with torch.no_grad():
        want = x + tmu(x, "incoming", mask, **w)
        got = _lib.host().multiplicative_update_residual(x, mask, False, 1e-5, _lib.PREC_IEEE, [w.get(n) for n in _lib.WEIGHT_NAMES])
    assert torch.equal(got, want)


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("shape", [(1, 3, 64, 2, 32), (1, 130, 130, 4, 32), (2, 40, 40, 2, 24)], ids=str)
def test_attention(shape, transposed):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import triangle_attention
    t, mask, res = util.attn_inputs(*shape, torch.bfloat16, seed=sum(shape))
    if transposed:
        res = res.transpose(1, 2).contiguous().transpose(1, 2)
    with torch.no_grad():
        want = res + triangle_attention(t["q"], t["k"], t["v"], t["bias"], mask)
        got = _lib.host().attention_residual(res, t["q"], t["k"], t["v"], t["bias"].expand(shape[0], 1, shape[3], shape[2], shape[2]),
                                             mask, _lib.PREC_IEEE)
    assert got.stride() == res.stride() and torch.equal(got, want)
