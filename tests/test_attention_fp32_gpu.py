"""The fp32-operand attention kernels at the edges of their tiles, against the fp64 oracle."""

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

SHAPES = [  # B, rows, residues, heads, head dim
    (1, 2, 3, 1, 4),          # three keys
    (1, 5, 63, 2, 32), (1, 5, 64, 2, 32), (1, 9, 129, 1, 32), (2, 21, 128, 2, 32),   # around one and two m tiles
    (1, 4, 97, 1, 6),         # head dim that is no multiple of four: element-wise copies
    (1, 11, 70, 2, 128),      # widest head dim, dbias in row chunks of unequal length
    (1, 3, 257, 1, 100),      # head dim padded to 128, a last tile of one row
]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("precision", ["ieee", "tf32"])
def test_against_oracle(shape, precision):
    from geometric_nn_ops_b200.triangle import triangle_attention
    t, mask, d_out = util.attn_inputs(*shape, torch.float32, seed=sum(shape))
    with util.matmul_precision(precision):
        out, grads = util.attn_fwd_bwd(triangle_attention, t, mask, None, d_out)
        torch.cuda.synchronize()
    o_ref, g_ref = util.attn_oracle(t, mask, None, d_out)
    cos_min, fro = util.ATTN_TOL[torch.float32, precision]
    if precision == "ieee":
        fro, worst = util.IEEE_REL_FRO, util.MAX_ABS_REL["ieee32"]
    else:
        worst = util.MAX_ABS_REL["tf32"]
    util.check_close("out", out, o_ref, cos_min, fro, worst)
    for name, val in grads.items():
        util.check_close("grad_" + name, val, g_ref[name], cos_min, fro, worst)


@pytest.mark.parametrize("shape", [(1, 6, 128, 4, 32), (1, 5, 101, 2, 64), (1, 4, 70, 2, 128)], ids=str)
def test_bias_is_added_in_one_rounding(shape):
    """A bias near 100 under every logit: exact fp32 products must not start from it.  fp32 numbers there lie 2^-17 apart, so that
    bias and mask in one rounding each leave a logit, and with it P, right to 2^-18 = 4e-6 each way; a sum that rounds
    after every term beside the bias was off by 1e-5 and more."""
    from geometric_nn_ops_b200.triangle import triangle_attention
    t, mask, d_out = util.attn_inputs(*shape, torch.float32, seed=2, keep=0.95)
    t["bias"] = t["bias"] * 0.5 + 100
    with util.matmul_precision("ieee"):
        out, grads = util.attn_fwd_bwd(triangle_attention, t, mask, None, d_out)
    o_ref, g_ref = util.attn_oracle(t, mask, None, d_out)
    util.check_close("out", out, o_ref, 1 - 1e-9, 4e-6)
    for name, val in grads.items():
        util.check_close("grad_" + name, val, g_ref[name], 1 - 1e-9, 4e-6)
