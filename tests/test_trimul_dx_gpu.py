"""The multiplicative update's gradients through both LayerNorms where the tiles of their kernels end: less than a tile of 128
pixels, half tiles, several entries, against the fp64 oracle with the repository's tolerances."""

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,precision", [(torch.bfloat16, "ieee"), (torch.float16, "ieee"), (torch.float32, "tf32")], ids=["bf16", "fp16", "tf32"])
@pytest.mark.parametrize("B,N", [(1, 8), (1, 16), (1, 24), (1, 40), (2, 8), (3, 24)])
@pytest.mark.parametrize("affine", [True, False], ids=["affine", "plain"])
def test_layernorm_gradients(dtype, precision, B, N, affine):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import triangle_multiplicative_update
    x, mask, w, d_out = util.trimul_inputs(B, N, 128, 128, dtype, seed=B * 100 + N)
    if not affine:
        for name in ("norm_in_weight", "norm_in_bias", "norm_out_weight", "norm_out_bias"):
            w.pop(name)
    else:
        w["norm_in_weight"] = w["norm_in_weight"] * torch.linspace(0.5, 2, 128, device="cuda").to(dtype)   # channels apart
        w["norm_out_weight"] = w["norm_out_weight"] * torch.linspace(2, 0.5, 128, device="cuda").to(dtype)
    with util.matmul_precision(precision):
        out, grads = util.trimul_fwd_bwd(triangle_multiplicative_update, x, mask, w, "outgoing", d_out)
    torch.cuda.synchronize()
    assert _lib.last_path() == "tcgen05"
    _, ref = util.trimul_oracle(x, mask, w, "outgoing", d_out)
    cos_min, fro = util.TRIMUL_TOL[dtype, precision]
    for name in grads:
        util.check_close("grad_" + name, grads[name], ref[name], cos_min, 2 * fro)   # (small sums: twice the tables' bound)
