"""triangle_multiplicative_update on B200: public wrapper and kernel-level entry.

Keeps the signature of the reference's public op
(``geometric_nn_ops_torch/triangle/_trimul.py:39-88``) and of its kernel-level
functions ``impl(x, direction, mask, *, eps, **weights)``
(``_kernels/trimul.py:404-422``, ``_reference/trimul.py:57-75``).  Unlike the
reference, whose kernels are forward-only and which sends every grad-requiring call
to eager torch, forward AND backward run in libtri_b200.so, called through the native extension
``csrc/torch_host.cpp``.  CPU tensors are rejected: there is no CPU implementation in this package.
"""

import torch

from .. import _lib, _precision

DIRECTIONS = ("outgoing", "incoming")
_DTYPES = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16, torch.float16: _lib.F16}


def is_outgoing(direction: str) -> bool:
    if direction not in DIRECTIONS:
        raise ValueError(f"direction must be one of {DIRECTIONS}, got {direction!r}")
    return direction == "outgoing"


def _aligned(t):
    """Contiguous and 16-byte aligned (TMA and the vector loads need it); copies only if it must."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def trimul_b200(x, direction="outgoing", mask=None, *, eps=1e-5, norm_in_weight=None, norm_in_bias=None,
                p_in_weight=None, p_in_bias=None, g_in_weight=None, g_in_bias=None, norm_out_weight=None,
                norm_out_bias=None, p_out_weight=None, p_out_bias=None, g_out_weight=None, g_out_bias=None):
    """Kernel-level triangle multiplicative update, forward and backward on the GPU.

    ``x`` is ``[*, N, N, C_z]``, ``mask`` broadcastable to ``[*, N, N]`` (1 = keep);
    ``p_in_weight`` / ``g_in_weight`` are the concatenated ``[a; b]`` projections.
    """
    outgoing = is_outgoing(direction)
    precision = _lib.PREC_IEEE
    if x.dtype is torch.float32 and _precision.torch_precision() == _precision.TF32:
        precision = _lib.PREC_TF32
    return _lib.host().multiplicative_update(x, mask, outgoing, eps, precision, [
        norm_in_weight, norm_in_bias, p_in_weight, p_in_bias, g_in_weight, g_in_bias, norm_out_weight, norm_out_bias,
        p_out_weight, p_out_bias, g_out_weight, g_out_bias])


def triangle_multiplicative_update(x, direction="outgoing", mask=None, norm_in_weight=None, norm_in_bias=None,
                                   p_in_weight=None, p_in_bias=None, g_in_weight=None, g_in_bias=None,
                                   norm_out_weight=None, norm_out_bias=None, p_out_weight=None, p_out_bias=None,
                                   g_out_weight=None, g_out_bias=None, eps=1e-5):
    """Triangle multiplicative update over a pair representation (reference signature).

    Returns ``[*, N, N, C_z]``.  fp32 matmuls follow
    ``torch.backends.cuda.matmul.fp32_precision``.  Dtypes without a kernel (fp64) are
    computed in fp32 and cast back.
    """
    is_outgoing(direction)
    kw = dict(norm_in_weight=norm_in_weight, norm_in_bias=norm_in_bias, p_in_weight=p_in_weight,
              p_in_bias=p_in_bias, g_in_weight=g_in_weight, g_in_bias=g_in_bias, norm_out_weight=norm_out_weight,
              norm_out_bias=norm_out_bias, p_out_weight=p_out_weight, p_out_bias=p_out_bias,
              g_out_weight=g_out_weight, g_out_bias=g_out_bias)
    if x.dtype in _DTYPES:
        return trimul_b200(x, direction, mask, eps=eps, **kw)
    out = trimul_b200(x.float(), direction, mask, eps=eps,
                      **{n: (None if t is None else t.float()) for n, t in kw.items()})
    return out.to(x.dtype)
