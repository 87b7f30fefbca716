"""triangle_attention on B200: public wrapper and kernel-level entry.

The public function keeps the signature and argument handling of the reference's
``geometric_nn_ops_torch/triangle/_triattn.py:23-106``; the kernel-level entry
``triangle_attention_b200`` stands where the reference has
``triangle_attention_triton`` (``_kernels/triangle_attention.py:1447-1484``).
All arithmetic happens in libtri_b200.so and the host work (broadcasts, allocation, autograd) in the native extension
``csrc/torch_host.cpp``; q/k/v/o are passed with their strides, so both the native ``[B, N_seq, N_res, H, D]`` layout
and the cuequivariance ``(B, N, H, S, D)`` layout (a transposed view) run without a copy.
"""

import ctypes

import torch

from .. import _lib, _precision

_DTYPES = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16, torch.float16: _lib.F16}


def _st4(t):
    s = t.stride()
    return (ctypes.c_int64 * 4)(s[0], s[1], s[2], s[3])


def _desc(q, k, v, o, bias, mask, scale, precision):
    """The C descriptor of a call, for callers of the C ABI."""
    B, S, N, H, D = q.shape
    d = _lib.TriAttnDesc()
    d.B, d.n_seq, d.n_res, d.H, d.D = B, S, N, H, D
    d.dtype = _DTYPES[q.dtype]
    d.precision = _lib.PREC_TF32 if precision == _precision.TF32 else _lib.PREC_IEEE
    d.scale = scale
    d.q_st, d.k_st, d.v_st, d.o_st = _st4(q), _st4(k), _st4(v), _st4(o)
    if bias is not None:
        bs = bias.stride()
        d.bias_st = (ctypes.c_int64 * 3)(bs[0], bs[2], bs[3])
    if mask is not None:
        ms = mask.stride()
        d.mask_st = (ctypes.c_int64 * 2)(ms[0], ms[1])
    return d


def _precision_code(t):
    if t.dtype is not torch.float32:      # 16-bit operands: the switch cannot change them
        return _lib.PREC_IEEE
    return _lib.PREC_TF32 if _precision.torch_precision() == _precision.TF32 else _lib.PREC_IEEE


def triangle_attention_b200(q, k, v, bias=None, mask=None, scale=None, dynamic=False, use_exp2=False,
                            return_aux=False):
    """Kernel-level entry on canonical 5-D shapes.

    ``q, k, v``: ``[B, N_seq, N_res, H, D]``; ``bias``: ``[B, 1, H, N_res, N_res]`` (batch may be
    a broadcast view); ``mask``: bool ``[B, N_seq, 1, 1, N_res]``, ``True`` keeps.
    ``dynamic`` and ``use_exp2`` are accepted for signature compatibility; the CUDA kernels
    take shapes at run time, so both settings give the same result.
    ``return_aux=True`` returns ``(out, lse, max)``: the log-sum-exp and the maximum of each query's
    logits, fp32 ``[B, N_seq, H, N_res, 1]`` (the cuequivariance ``(B, N, H, Q, 1)`` layout), not differentiable.
    ``lse`` is exact.  ``max`` is the reference point the kernel used for the exponentials: the exact row maximum on
    the CUDA-core path; on the tensor-core path a value between ``max - 8 ln 2`` and ``max``.  That path serves 16-bit
    types, and fp32 with TF32 products (head dim up to 32) from 2e7 logits, B * N_seq * H * N_res**2, on; fp32 at "ieee" is
    always exact.  (The reference's kernels
    do not expose them and its cuequivariance shim raises for ``return_aux``,
    ``cuequivariance_ops_torch/triangle_attention.py:34-38``; these kernels write them anyway.)
    """
    return _lib.host().attention(q, k, v, bias, mask, scale, _precision_code(q), return_aux)


def triangle_attention(q, k, v, bias=None, mask=None, scale=None, dynamic=False, use_exp2=False, return_aux=False):
    """Triangle attention with the reference's (cuequivariance-compatible) signature.

    Args:
        q, k, v: ``[..., N_seq, N_res, H, D]``; rank 4, 5 or 6 (leading dims fold into one batch).
        bias: broadcastable to ``[B, 1, H, N_res, N_res]``, or ``None``.
        mask: bool, ``True`` keeps; broadcastable to ``[B, N_seq, 1, 1, N_res]``, or ``None``.
        scale: softmax scale, default ``D ** -0.5``.

    Returns a tensor of q's shape and dtype; with ``return_aux=True`` also the log-sum-exp and the
    maximum of every query's logits (fp32, ``[B, N_seq, H, N_res, 1]``).  The maximum is exact for fp32 at "ieee"; for
    16-bit types and TF32 it may lie up to ``8 ln 2`` below it (see :func:`triangle_attention_b200`).  fp32 matmuls follow
    ``torch.backends.cuda.matmul.fp32_precision``.
    """
    if mask is not None and mask.dtype != torch.bool:
        raise ValueError(f"mask must be bool (keep=True/mask=False), got {mask.dtype}")

    if q.dtype in _DTYPES:
        return _lib.host().attention(q, k, v, bias, mask, scale, _precision_code(q), return_aux)
    # a dtype without a kernel (fp64) is computed in fp32 and cast back
    cast = lambda t: None if t is None else t.float()  # noqa: E731
    res = triangle_attention(cast(q), cast(k), cast(v), cast(bias), mask, scale, return_aux=return_aux)
    return (res[0].to(q.dtype), *res[1:]) if return_aux else res.to(q.dtype)
