"""Rows masked through the bias (large finite values, the type's lowest, infinity) against softmax over fp32 logits.

The logits are the reference's: fp32 sums, so that a term beside a bias of -1e9 is lost to rounding (geometric_nn_ops_torch/
triangle/_reference/triangle_attention.py:28-44 adds bias and mask in fp32).  Softmax, products and gradients follow in fp64.
"""

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

SHAPES = [(1, 5, 136, 2, 32), (1, 4, 301, 2, 32),   # three rows per bias tile, even and odd lengths
          (1, 2, 136, 2, 32), (1, 3, 136, 2, 64)]   # two rows; a wide head
LEVELS = {torch.bfloat16: [-1e8, -6.9e7, -1e9, torch.finfo(torch.bfloat16).min, float("-inf"), 1e8],
          torch.float16: [-30000.0, torch.finfo(torch.float16).min, float("-inf")],
          torch.float32: [-1e8, -1e9, torch.finfo(torch.float32).min, float("-inf"), 1e8]}
CASES = [(dtype, "ieee", level) for dtype, levels in LEVELS.items() for level in levels] + [(torch.float32, "tf32", float("-inf"))]


def _reference(t, mask, d_out):
    scale = t["q"].shape[-1] ** -0.5
    heads = lambda x: x.transpose(2, 3)  # noqa: E731
    q, k, v, do = (heads(x).double() for x in (t["q"], t["k"], t["v"], d_out))
    x = (q @ k.transpose(-1, -2) * scale).float() + t["bias"].float() + 1e9 * (mask.float() - 1)
    p = torch.softmax(x.double(), -1)
    dp = do @ v.transpose(-1, -2)
    ds = p * (dp - (dp * p).sum(-1, keepdim=True))
    return heads(p @ v), {"q": heads(ds @ k) * scale, "k": heads(ds.transpose(-1, -2) @ q) * scale, "v": heads(p.transpose(-1, -2) @ do),
                          "bias": ds.sum(1, keepdim=True)}


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("dtype,precision,level", CASES, ids=lambda v: str(v).replace("torch.", ""))
def test_rows_masked_by_the_bias(shape, dtype, precision, level):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import triangle_attention
    n = shape[2]
    t, mask, d_out = util.attn_inputs(*shape, dtype, seed=sum(shape), keep=0.95)
    t["q"] *= 0.5          # logits of q and k within 3: beside the level they are lost, whatever the order of the sum
    if level % 64 != 32:   # (halfway between two fp32 numbers at 1e9 the order of the sum decides)
        mask[0, 1] = False     # a row of the pair tensor with no key at all
    b = t["bias"]
    if level != float("-inf"):
        b[..., 3, :] = level                     # a whole row
        b[..., n - 1, :] = level
    b[..., 7, :64] = level                       # the first key step
    b[..., 40, :-1] = level                      # all but the last key ...
    b[..., 41, 1:] = level                       # ... but the first
    b[..., 70:75, ::2] = level
    mask[0, 0, ..., -1] = True
    with util.matmul_precision(precision):
        out, grads = util.attn_fwd_bwd(triangle_attention, t, mask, None, d_out)
    torch.cuda.synchronize()
    assert _lib.last_path() == ("simt" if dtype == torch.float32 else "tcgen05")
    o_ref, g_ref = _reference(t, mask, d_out)
    cos_min, fro = util.ATTN_TOL[dtype, precision]
    util.check_close("out", out, util.f64(o_ref), cos_min, fro)
    for name, val in grads.items():
        util.check_close("grad_" + name, val, util.f64(g_ref[name]), cos_min, fro)
