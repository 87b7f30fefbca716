"""Forward-mode derivatives: the kernels have none and say so; what attention_pair_bias leaves to torch keeps them."""

import pytest
import torch
import torch.autograd.forward_ad as fwd

from tests import util

pytestmark = pytest.mark.gpu


def _dual(t):
    return fwd.make_dual(t, torch.ones_like(t))


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("which", ["q", "v", "bias"])
def test_attention_refuses(which, grad):
    from geometric_nn_ops_b200.triangle import triangle_attention
    t, mask, _ = util.attn_inputs(1, 4, 64, 2, 32, torch.bfloat16, seed=1)
    with fwd.dual_level(), torch.set_grad_enabled(grad):
        t[which] = _dual(t[which].requires_grad_(grad))
        with pytest.raises(NotImplementedError, match="forward-mode"):
            triangle_attention(t["q"], t["k"], t["v"], t["bias"], mask)


@pytest.mark.parametrize("which", ["x", "p_in_weight"])
def test_update_refuses(which):
    from geometric_nn_ops_b200.triangle import trimul_b200
    x, mask, w, _ = util.trimul_inputs(1, 16, 128, 128, torch.bfloat16, seed=1)
    with fwd.dual_level():
        if which == "x":
            x = _dual(x)
        else:
            w[which] = _dual(w[which])
        with pytest.raises(NotImplementedError, match="forward-mode"):
            trimul_b200(x, "outgoing", mask, **w)


def test_pair_stack_refuses():
    from geometric_nn_ops_b200 import pairstack
    z, mask = torch.randn(1, 16, 16, 128, device="cuda").bfloat16(), torch.ones(1, 16, 16, device="cuda").bfloat16()
    blocks = [pairstack.make_block_weights(0, dtype=torch.bfloat16, device="cuda")]
    with fwd.dual_level(), pytest.raises(NotImplementedError, match="forward-mode"):
        pairstack.pair_stack(_dual(z), mask, blocks)


def test_pair_bias_gate_keeps_its_tangent():
    """The gate and output projections are torch's: out = Wo (o * sigmoid(Wg s)) with a tangent on s."""
    from geometric_nn_ops_b200.triangle import attention_pair_bias
    g = torch.Generator(device="cuda").manual_seed(0)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.float32).bfloat16()  # noqa: E731
    s, q, k, v, z = rn(1, 64, 96), rn(1, 4, 64, 24), rn(1, 4, 64, 24), rn(1, 4, 64, 24), rn(1, 64, 64, 128)
    w = {"proj_g_weight": rn(96, 96) * 0.1, "proj_o_weight": rn(96, 96) * 0.1, "proj_z_weight": rn(4, 128) * 0.1, "ln_z_weight": rn(128)}
    with fwd.dual_level():
        got = fwd.unpack_dual(attention_pair_bias(_dual(s), q, k, v, z, **w)[0]).tangent
        with pytest.raises(NotImplementedError, match="forward-mode"):
            attention_pair_bias(s, _dual(q), k, v, z, **w)
    step = torch.full_like(s, 1.0).double()
    eye = dict(w, proj_o_weight=torch.eye(96, device="cuda").bfloat16())
    pre = s.double() @ w["proj_g_weight"].double().T
    core = attention_pair_bias(s, q, k, v, z, **eye)[0].double() / pre.sigmoid()     # o
    slope = pre.sigmoid() * (1 - pre.sigmoid()) * (step @ w["proj_g_weight"].double().T)
    want = (core * slope) @ w["proj_o_weight"].double().T
    assert (got.double() - want).norm() / want.norm() < 2e-2      # a handful of bf16 roundings
