"""The CUDA-core multiplicative update at the edges of its kernels' tiles and dispatch, against the fp64 oracle."""

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

CASES = [  # B, N, C, Ch
    (1, 9, 4, 4),         # the narrowest rows of the fused kernels
    (1, 65, 128, 128),    # the contraction's r axis in four parts of unequal length, last tiles of one pixel
    (1, 150, 128, 64),    # 8 x 8 tiles over the whole r axis, two channel groups per CTA
    (3, 21, 68, 132),     # channels that are no multiple of a 64-wide block
    (2, 11, 30, 20),      # channels that are no multiple of four: one stage per kernel
    (1, 10, 264, 40),     # rows too wide for the fused kernels
    (1, 68, 128, 128), (1, 69, 128, 128),   # output stage in tiles of 32 pixels, of 64
    (1, 33, 132, 256), (1, 60, 256, 128),   # rows of more than 128 channels, tiles of 32 and of 64
]


@pytest.mark.parametrize("direction", ["outgoing", "incoming"])
@pytest.mark.parametrize("case", CASES, ids=str)
def test_against_oracle(case, direction):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.triangle import triangle_multiplicative_update as tmu
    B, N, C, Ch = case
    x, mask, w, d_out = util.trimul_inputs(B, N, C, Ch, torch.float32, seed=N + C, biases=True)
    with util.matmul_precision("ieee"):
        out, grads = util.trimul_fwd_bwd(tmu, x, mask, w, direction, d_out)
        with torch.no_grad():
            infer = tmu(x, direction, mask, **w)
    assert _lib.last_path() == "simt" and torch.equal(infer, out)
    o_ref, g_ref = util.trimul_oracle(x, mask, w, direction, d_out)
    util.check_close("out", out, o_ref, 1 - 1e-9, util.IEEE_REL_FRO, 1e-4)
    for name, val in grads.items():
        util.check_close("grad_" + name, val, g_ref[name], 1 - 1e-9, util.IEEE_REL_FRO, 1e-4)
