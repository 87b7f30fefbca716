"""Where the tensor-core attention forward takes its key-mask terms from: the mask bytes (short calls) or terms made before (long ones)."""

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu


def _ta():
    from geometric_nn_ops_b200.triangle import triangle_attention
    return triangle_attention


def _moved(mask, off):
    """The same mask `off` bytes behind an aligned address."""
    flat = torch.empty(mask.numel() + off, dtype=mask.dtype, device=mask.device)
    return flat[off:].view(mask.shape).copy_(mask)


# rows of a length of 0 to 3 modulo 4, so that rows start at every offset in a word; last key steps of 1, 2, 62 and 64 keys
@pytest.mark.parametrize("n,dim", [(257, 32), (322, 32), (191, 32), (320, 32), (257, 64), (254, 64)], ids=str)
def test_mask_bytes_at_every_alignment(n, dim):
    from geometric_nn_ops_b200 import _lib
    t, mask, _ = util.attn_inputs(1, 20, n, 2, dim, torch.bfloat16, seed=n, keep=0.5)
    mask[0, 3] = False
    mask[0, 5] = torch.arange(n, device="cuda") == n - 1
    with torch.no_grad():
        x = torch.einsum("bsqhd,bskhd->bshqk", t["q"].double() * dim ** -0.5, t["k"].double()) + t["bias"].double() + 1e9 * (mask.double() - 1)
        want = torch.einsum("bshqk,bskhd->bsqhd", torch.softmax(x, -1), t["v"].double())
        want[0, 3] = t["v"].double()[0, 3].mean(0)       # -1e9 swallows the logits of a row without a kept key
        base = _ta()(t["q"], t["k"], t["v"], t["bias"], mask)
        assert _lib.last_path() == "tcgen05"
        util.check_close("out", base, util.f64(want), *util.ATTN_TOL[torch.bfloat16, "ieee"], util.MAX_ABS_REL[torch.bfloat16])
        for off in (1, 2, 3, 5):
            assert torch.equal(_ta()(t["q"], t["k"], t["v"], t["bias"], _moved(mask, off)), base)


def test_terms_made_before():
    """2.8e8 logits, above the line, against the same rows in calls below it: a row's result does not depend on the others."""
    t, mask, _ = util.attn_inputs(1, 546, 358, 4, 32, torch.bfloat16, seed=2)
    with torch.no_grad():
        out = _ta()(t["q"], t["k"], t["v"], t["bias"], mask)
        for s in (0, 270, 543):
            part = _ta()(*(t[k][:, s:s + 3] for k in ("q", "k", "v")), t["bias"], mask[:, s:s + 3])
            assert torch.equal(part, out[:, s:s + 3])
