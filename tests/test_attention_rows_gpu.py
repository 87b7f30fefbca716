"""The row-sharing forward kernel and the padded tensor-core path (odd lengths, head dims below a tile) at their edges."""

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

SHAPES = [  # B, rows, residues, heads, head dim
    (1, 57, 57, 4, 32),      # just above the smallest ragged problem; one key step, the last triple complete
    (2, 40, 65, 4, 32),      # a second key step of one key, two rows in the last triple, two batch entries
    (1, 301, 48, 2, 32),     # several items per CTA, one key step each
    (1, 7, 301, 4, 32),      # five key steps, 45 queries in the last block, one row in the last triple
    (1, 3, 520, 2, 24),      # head dim padded to 32, one triple
    (1, 2, 385, 4, 48),      # head dim padded to 64, two rows
    (1, 5, 193, 4, 64), (1, 16, 200, 4, 8),
]


def _ta():
    from geometric_nn_ops_b200.triangle import triangle_attention
    return triangle_attention


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=str)
def test_against_oracle(shape, dtype):
    from geometric_nn_ops_b200 import _lib
    t, mask, d_out = util.attn_inputs(*shape, dtype, seed=sum(shape))
    out, grads = util.attn_fwd_bwd(_ta(), t, mask, None, d_out)
    torch.cuda.synchronize()
    assert _lib.last_path() == "tcgen05"
    o_ref, g_ref = util.attn_oracle(t, mask, None, d_out)
    cos_min, fro = util.ATTN_TOL[dtype, "ieee"]
    util.check_close("out", out, o_ref, cos_min, fro, util.MAX_ABS_REL[dtype])
    for name, val in grads.items():
        util.check_close("grad_" + name, val, g_ref[name], cos_min, fro, util.MAX_ABS_REL[dtype])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=str)
@pytest.mark.parametrize("starts", [(5, 70, 300), (17, 63, 64), (200, 201, 447)], ids=str)
def test_rows_that_outgrow_their_reference(dtype, starts):
    """Logits that climb by up to 100 at chosen keys, a fully masked row, a row whose first 300 keys are masked."""
    t, mask, _ = util.attn_inputs(1, 8, 512, 4, 32, dtype, seed=5)
    g = torch.Generator().manual_seed(9)
    for i, k in enumerate(starts):
        t["bias"][..., k:] += (torch.rand(1, 1, 4, 512, 1, generator=g) * 70 + (30 if i else 0)).to(dtype).cuda()
    mask[0, 2, ..., :300] = False
    with torch.no_grad():
        out, lse, top = _ta()(t["q"], t["k"], t["v"], t["bias"], mask, return_aux=True)
    x = torch.einsum("bsqhd,bskhd->bshqk", t["q"].double() * 32 ** -0.5, t["k"].double()) + t["bias"].double()
    x = x + 1e9 * (mask.double() - 1)
    want = torch.einsum("bshqk,bskhd->bsqhd", torch.softmax(x, -1), t["v"].double())
    util.check_close("out", out, util.f64(want), *util.ATTN_TOL[dtype, "ieee"], util.MAX_ABS_REL[dtype])
    assert (lse[..., 0].double() - x.logsumexp(-1)).abs().max() < 1e-3
    gap = x.amax(-1) - top[..., 0].double()
    assert gap.min() > -1e-3 and gap.max() < 8 * 0.6932        # the reported maximum may lag by up to 8 ln 2
    mask[0, 1] = False
    with torch.no_grad():
        out = _ta()(t["q"], t["k"], t["v"], t["bias"] * 0.01, mask)
    assert (out[0, 1].float() - t["v"][0, 1].float().mean(0)).abs().max() <= 2e-2
