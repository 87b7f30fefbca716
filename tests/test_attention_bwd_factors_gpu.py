"""Row constants that reach the attention backward through the products: what a factor can hold, and rows that go without.

A row (batch, row, head) leaves the factors when one of its queries has a maximum beyond 256, or, in fp16, a delta beyond 31 or
a constant beyond 6e4; fp16 holds delta in steps of 2^-48, so that small upstream gradients keep their digits.
The reference is softmax over fp64 logits of the rounded inputs.  P and dS are rounded to the operand type before their
products, so a gradient is off by about half a unit in the last place of each term: 2^-9 (bf16), 2^-12 (fp16), and at most
four times that is allowed in the 2-norm.
"""

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu


def _reference(t, mask, d_out, scale):
    heads = lambda x: x.transpose(2, 3).double()  # noqa: E731
    q, k, v, do = (heads(x) for x in (t["q"], t["k"], t["v"], d_out))
    x = q @ k.transpose(-1, -2) * scale + t["bias"].double()
    p = torch.softmax(x.masked_fill(~mask.expand(x.shape), float("-inf")), -1)
    dp = do @ v.transpose(-1, -2)
    ds = p * (dp - (dp * p).sum(-1, keepdim=True))
    back = lambda x: x.transpose(2, 3)  # noqa: E731
    return {"q": back(ds @ k) * scale, "k": back(ds.transpose(-1, -2) @ q) * scale, "v": back(p.transpose(-1, -2) @ do),
            "bias": ds.sum(1, keepdim=True)}


# lengths: one query tile, one and a half key blocks, an odd number of tiles, rows that are no multiple of eight
@pytest.mark.parametrize("shape", [(1, 3, 64, 2, 32), (2, 4, 136, 3, 32), (1, 9, 320, 2, 32), (1, 31, 103, 2, 32), (1, 5, 136, 2, 16), (1, 3, 200, 2, 64)],
                         ids=str)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("d_scale", [2.0 ** -13, 1.0, 64.0], ids=["small", "one", "large"])
@pytest.mark.parametrize("shift", [0.0, 240.0, 300.0])
def test_backward(shape, dtype, d_scale, shift):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import triangle_attention
    t, mask, d_out = util.attn_inputs(*shape, dtype, seed=sum(shape), keep=0.9)
    # a shift of whole rows of the bias moves the maximum and nothing else; every third query, so that rows mix
    t["bias"][..., ::3, :] = (t["bias"][..., ::3, :].float() * (1 if shift == 0 else 0) + shift).to(dtype)
    d_out = (d_out.float() * d_scale).to(dtype)
    scale = 0.2
    out, grads = util.attn_fwd_bwd(triangle_attention, t, mask, scale, d_out)
    torch.cuda.synchronize()
    assert _lib.last_path() == "tcgen05"
    limit = 4 * (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12)
    for name, want in _reference(t, mask, d_out, scale).items():
        if dtype == torch.float16 and d_scale < 1 and name in "qk":
            continue   # dS is an fp16 operand of these products and below its normal range
        got = grads[name].double()
        assert torch.isfinite(got).all(), name
        slack = 2.0 ** -25 * want.numel() ** 0.5 / float(want.norm()) if dtype == torch.float16 else 0.0   # fp16's smallest step
        err = float((got - want).norm() / want.norm())
        assert err <= limit + slack, f"{name}: {err:.2e} > {limit + slack:.2e}"


# odd numbers of 64-query tiles: the last one's dQ product has no partner, and its own columns
@pytest.mark.parametrize("n", [136, 192, 301, 320, 64])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
def test_unpaired_last_tile(n, dtype):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import triangle_attention
    t, mask, d_out = util.attn_inputs(1, 96, n, 4, 32, dtype, seed=n, keep=0.9)
    _, grads = util.attn_fwd_bwd(triangle_attention, t, mask, 0.2, d_out)
    torch.cuda.synchronize()
    assert _lib.last_path() == "tcgen05"
    limit = 4 * (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12)
    for name, want in _reference(t, mask, d_out, 0.2).items():
        err = float((grads[name].double() - want).norm() / want.norm())
        assert err <= limit, f"{name}: {err:.2e} > {limit:.2e}"
    for _ in range(40):
        _, again = util.attn_fwd_bwd(triangle_attention, t, mask, 0.2, d_out)
        for name, first in grads.items():
            assert torch.equal(again[name], first), name
