"""The phases of the row-sharded multiplicative update on one GPU: the shards one after the other, the exchanges by torch.

Against the whole update on the same inputs.  The forward's arithmetic per pixel is the same; weight gradients are sums over the
shards instead of one split-K sum, and the bf16 gradients that the phases hand on are rounded alike.
"""

import ctypes

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu


class _Shard:
    def __init__(self, x, mask, w, precision):
        from geometric_nn_ops_b200 import _lib, sharded
        self.lib, self.phase = _lib.load(), sharded._phase
        B, R, N, C = x.shape
        self.d = _lib.TriMulShardDesc(B, R, N, C, C, sharded._DTYPES[x.dtype], precision, 1e-5)
        size = lambda f: torch.empty(f(ctypes.byref(self.d)), dtype=torch.uint8, device="cuda")  # noqa: E731
        self.saved, self.prep = size(self.lib.tri_mul_shard_saved_bytes), size(self.lib.tri_mul_shard_prep_bytes)
        self.grads = {n: torch.full(t.shape, float("nan"), device="cuda") for n, t in w.items()}
        self.keep = [x, mask]
        self.w, self.g = _lib.TriMulWeights(), _lib.TriMulWeightGrads()
        for n, t in w.items():
            setattr(self.w, _lib.abi_field(n), t.data_ptr())
            setattr(self.g, _lib.abi_field(n), self.grads[n].data_ptr())
        b = self.bufs = _lib.TriMulShardBufs()
        b.x, b.mask, b.w, b.g = x.data_ptr(), mask.data_ptr(), ctypes.pointer(self.w), ctypes.pointer(self.g)
        b.saved, b.prep, b.prep_ready = self.saved.data_ptr(), self.prep.data_ptr(), 0
        self.plane = (B, C, R, N)

    def run(self, phase, **tensors):
        for name, t in tensors.items():
            assert t.is_contiguous()
            self.keep.append(t)
            setattr(self.bufs, name, t.data_ptr())
        self.phase(self.lib, self.d, phase, self.bufs, torch.device("cuda", torch.cuda.current_device()))
        self.bufs.prep_ready = 1     # every later phase is a call whose first kernel is the phase's own


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=str)
def test_tensors_off_16_bytes_are_refused(dtype):
    from geometric_nn_ops_b200 import _lib
    x, mask, w, d_out = util.trimul_inputs(1, 32, 128, 128, dtype, seed=1)
    s = _Shard(x[:, :16].contiguous(), mask[:, :16].contiguous(), w, _lib.PREC_TF32)
    room = torch.zeros(1 << 24, dtype=torch.uint8, device="cuda")
    launches = _lib.launch_count()
    names = {_lib.PHASE_PROJECT: ["x", "saved", "prep", "a_cm", "b_cm"] + (["mask"] if dtype == torch.float32 else []),
             _lib.PHASE_OUTPUT: ["saved", "t_cm", "out"], _lib.PHASE_OUTPUT_BWD: ["saved", "t_cm", "d_out", "dt_cm"],
             _lib.PHASE_PROJECT_BWD: ["x", "mask", "saved", "a_cm", "b_cm", "dx"]}
    for name in ("a_cm", "b_cm", "t_cm", "out", "d_out", "dt_cm", "dx"):
        setattr(s.bufs, name, room.data_ptr())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for phase, tensors in names.items():
        for name in tensors + ["ws"]:
            aligned, off = (0, 8) if name == "ws" else (getattr(s.bufs, name), 0)
            if name != "ws":
                setattr(s.bufs, name, aligned + 8)
            at = ctypes.c_void_p(room.data_ptr() + off)
            assert s.lib.tri_mul_shard_phase(ctypes.byref(s.d), phase, ctypes.byref(s.bufs), at, room.numel() - 16, stream) == -1, (phase, name)
            if name != "ws":
                setattr(s.bufs, name, aligned)
    assert _lib.launch_count() == launches


@pytest.mark.parametrize("direction", ["outgoing", "incoming"])
@pytest.mark.parametrize("dtype,precision,B,n", [(torch.bfloat16, "ieee", 1, 64), (torch.float16, "ieee", 2, 48), (torch.float32, "tf32", 1, 48),
                                                 (torch.bfloat16, "ieee", 1, 264)], ids=lambda v: str(v).replace("torch.", ""))
def test_phases_of_two_shards(dtype, precision, B, n, direction):
    from geometric_nn_ops_b200 import _lib
    from geometric_nn_ops_b200.gemm import bgemm
    from geometric_nn_ops_b200.triangle import trimul_b200
    x, mask, w, d_out = util.trimul_inputs(B, n, 128, 128, dtype, seed=n, biases=True)
    with util.matmul_precision(precision):
        want, g_want = util.trimul_fwd_bwd(trimul_b200, x, mask, w, direction, d_out)
    code = _lib.PREC_TF32 if precision == "tf32" else _lib.PREC_IEEE
    R = n // 2
    part = lambda t, r, dim=1: t.narrow(dim, r * R, R).contiguous()  # noqa: E731
    shards = [_Shard(part(x, r), part(mask, r), w, code) for r in range(2)]
    new = lambda s: torch.full(s.plane, float("nan"), dtype=dtype, device="cuda")  # noqa: E731
    rows = lambda ts: torch.cat(ts, 2).reshape(B * 128, n, n)  # noqa: E731
    ab = []
    for s in shards:
        ab.append((new(s), new(s)))
        s.run(_lib.PHASE_PROJECT, a_cm=ab[-1][0], b_cm=ab[-1][1])
    a, b = rows([p[0] for p in ab]), rows([p[1] for p in ab])
    inc = direction == "incoming"
    t = bgemm(a, b, a_mn_major=inc, b_mn_major=inc).reshape(B, 128, n, n)
    outs, dts = [], []
    for r, s in enumerate(shards):
        outs.append(torch.full_like(part(x, r), float("nan")))
        s.run(_lib.PHASE_OUTPUT, t_cm=part(t, r, 2), out=outs[-1])
    for r, s in enumerate(shards):
        dts.append(new(s))
        s.run(_lib.PHASE_OUTPUT_BWD, d_out=part(d_out, r), dt_cm=dts[-1])
    dt = rows(dts)
    if inc:
        da, db = bgemm(b, dt), bgemm(a, dt, b_mn_major=True)
    else:
        da, db = bgemm(dt, b, b_mn_major=True), bgemm(dt, a, a_mn_major=True, b_mn_major=True)
    dxs = []
    for r, s in enumerate(shards):
        dxs.append(torch.full_like(part(x, r), float("nan")))
        s.run(_lib.PHASE_PROJECT_BWD, a_cm=part(da.reshape(B, 128, n, n), r, 2), b_cm=part(db.reshape(B, 128, n, n), r, 2), dx=dxs[-1])
    torch.cuda.synchronize()
    rel = lambda got, ref: float((got.detach().double() - ref.detach().double()).norm() / ref.detach().double().norm())  # noqa: E731
    assert rel(torch.cat(outs, 1), want) <= 1e-3
    # one unit in the last place of what is rounded between the phases, and of the result
    limit = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
    assert rel(torch.cat(dxs, 1), g_want["x"]) <= limit
    for name in w:
        assert rel(shards[0].grads[name] + shards[1].grads[name], g_want[name]) <= limit, name
