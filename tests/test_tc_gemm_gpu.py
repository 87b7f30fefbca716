"""The tcgen05 batched GEMM against an fp64 matmul of the same (rounded) inputs."""

import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [  # batch, M, N, K
    (1, 128, 128, 64), (1, 128, 256, 128), (3, 256, 512, 192), (2, 200, 136, 72), (4, 768, 768, 768),
    (1, 64, 40, 24),
    (40, 512, 512, 128), (80, 456, 504, 72), (40, 504, 488, 448),   # pairs of SMs: whole and ragged tiles, more stages than there are
    (2, 208, 208, 208), (2, 136, 264, 64), (1, 384, 384, 384), (1, 128, 520, 128),   # tiles narrower than 256 columns, pieces of 8 and 16
]


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (True, True), (False, True), (True, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=str)
@pytest.mark.parametrize("case", CASES, ids=str)
def test_bgemm(case, dtype, a_mn, b_mn):
    from geometric_nn_ops_b200.gemm import bgemm
    batch, M, N, K = case
    g = torch.Generator().manual_seed(M + N + K)
    a = torch.randn(batch, M, K, generator=g).to(dtype).cuda()
    b = torch.randn(batch, N, K, generator=g).to(dtype).cuda()
    want = torch.matmul(a.double(), b.double().transpose(1, 2))
    a_in = a.transpose(1, 2).contiguous() if a_mn else a
    b_in = b.transpose(1, 2).contiguous() if b_mn else b
    got32 = bgemm(a_in, b_in, a_mn_major=a_mn, b_mn_major=b_mn, out_dtype=torch.float32, check=True)
    rel = ((got32.double() - want).norm() / want.norm()).item()
    assert rel < (1e-3 if dtype == torch.float32 else 1e-5), rel   # tf32 drops 13 mantissa bits; 16-bit products are exact
    got = bgemm(a_in, b_in, a_mn_major=a_mn, b_mn_major=b_mn, check=True)
    assert got.dtype == dtype
    assert torch.equal(got, got32.to(dtype))


# whole tiles; an M that is no multiple of four, whose rows are stored one by one; rows of an odd length; one tile of 256 x 256 for 148 pairs
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (True, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=str)
@pytest.mark.parametrize("case", [(40, 512, 512, 576), (40, 509, 512, 584), (40, 510, 511, 600), (148, 256, 256, 640)], ids=str)
def test_pairs_of_sms(case, dtype, a_mn, b_mn):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.gemm import bgemm
    batch, M, N, K = case
    if (a_mn and M % 8 != 0) or (b_mn and N % 8 != 0):
        pytest.skip("rows of such operands start on 16-byte boundaries")
    g = torch.Generator().manual_seed(M + N + K)
    a = torch.randn(batch, M, K, generator=g).to(dtype).cuda()
    b = torch.randn(batch, N, K, generator=g).to(dtype).cuda()
    want = torch.matmul(a.double(), b.double().transpose(1, 2))
    a, b = (t.transpose(1, 2).contiguous() if mn else t for t, mn in ((a, a_mn), (b, b_mn)))
    _lib.profile_enable(True)
    got = bgemm(a, b, a_mn_major=a_mn, b_mn_major=b_mn, check=True)
    names = set(_lib.profile_summary())
    _lib.profile_enable(False)
    assert names == {"tc_bgemm_pair"}, names
    rel = ((got.double() - want).norm() / want.norm()).item()
    # tf32 drops 13 mantissa bits of either factor; the results' own rounding otherwise
    assert rel < {torch.float32: 1e-3, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype], rel


@pytest.mark.parametrize("dtype,K,pair", [(torch.bfloat16, 512, False), (torch.bfloat16, 576, True), (torch.float16, 520, True), (torch.float32, 352, False),
                                          (torch.float32, 384, True)], ids=str)
def test_short_sums_stay_on_single_sms(dtype, K, pair):
    """A pair's tile gains where its products outlast the stores of the tile before."""
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.gemm import bgemm
    a, b = torch.ones(40, 512, K, dtype=dtype, device="cuda"), torch.ones(40, 512, K, dtype=dtype, device="cuda")
    _lib.profile_enable(True)
    got = bgemm(a, b)
    names = set(_lib.profile_summary())
    _lib.profile_enable(False)
    assert names == {"tc_bgemm_pair" if pair else "tc_bgemm"}
    assert bool((got == float(K)).all())
