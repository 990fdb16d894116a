"""Host side of the FLARE gather-scatter mixer: the reference's Python surface over the C ABI.

``flare_multihead_mixer(q, k, v)`` has the signature and meaning of the function
of the same name in the reference's README.md:37-53 (the two SDPA calls inside
``FLARE.forward``, pdebench/models/flare.py:136-138 and
lra/models/backends.py:603-606) and is differentiable.  ``flare_gather`` and
``flare_scatter`` expose the two calls separately for callers that touch the
latents in between (pdebench/models/flare_ablations.py:93-132).

PyTorch supplies device memory, streams and autograd bookkeeping; all
arithmetic happens in libflare_b200.so.  CPU tensors are rejected: there is no
fallback path.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional, Tuple

import torch

from . import _cabi
from ._cabi import FlareProblem, check, lib, native

ops = torch.ops.flare_b200

__all__ = [
    "flare_multihead_mixer", "flare_gather", "flare_scatter",
    "mixer_forward", "mixer_backward", "gather_forward", "gather_backward", "scatter_forward", "scatter_backward",
    "make_problem", "set_kernel_path", "device_status", "pass_counts",
]


def set_kernel_path(path: str) -> str:
    """'auto' (tensor-core kernels where the shape allows) or 'simt'; returns the previous one."""
    code = {"auto": 0, "simt": 1, "tc_exact": 2}[path]
    prev = lib.flare_set_path(code)
    return {0: "auto", 1: "simt", 2: "tc_exact"}[prev]


def device_status(clear: bool = True) -> int:
    """Status word of the current device (synchronises): non-zero if a tensor-core kernel gave up on a
    bounded wait since the word was last cleared, in which case that kernel's output is not valid."""
    out = C.c_int(0)
    check(lib.flare_device_status(C.byref(out), 1 if clear else 0), "flare_device_status")
    return out.value


def pass_counts():
    """(tensor-core passes, fp32-kernel passes) enqueued by this process so far."""
    tc, simt = C.c_longlong(0), C.c_longlong(0)
    check(lib.flare_pass_counts(C.byref(tc), C.byref(simt)), "flare_pass_counts")
    return tc.value, simt.value


def _need_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise RuntimeError("flare_b200 runs on CUDA tensors only (sm_100a); got a CPU tensor")


def _tok(t: torch.Tensor) -> torch.Tensor:
    """A [B,H,N,D] tensor the kernels can address: unit stride on D, 16-byte aligned rows, no broadcast
    (stride 0) dimension -- a TMA tensor map cannot describe one."""
    e = t.element_size()
    ok = t.stride(-1) == 1 and t.data_ptr() % 16 == 0 and \
        all((s * e) % 16 == 0 and (s != 0 or n == 1) for s, n in zip(t.stride()[:-1], t.shape[:-1]))
    return t if ok else t.contiguous()


def _q3(q: torch.Tensor) -> Tuple[torch.Tensor, bool]:
    """q as [H,M,D] (shared latents) or [B,H,M,D]; an expand()-ed batch is folded back."""
    if q.dim() == 4 and q.stride(0) == 0:
        q = q[0]
    if q.dim() not in (3, 4):
        raise ValueError(f"q must be [H,M,D] or [B,H,M,D], got {tuple(q.shape)}")
    return _tok(q), q.dim() == 4


def make_problem(q, k, scale: float, n_splits: int = 0, v=None, y=None, dy=None, dk=None, dv=None,
                 dropout_p: float = 0.0, dropout_seed: int = 0) -> FlareProblem:
    B, H, N, D = k.shape
    if q.dim() == 3:
        Hq, M, Dq = q.shape
        qs = (0, q.stride(0), q.stride(1))
    else:
        Bq, Hq, M, Dq = q.shape
        if Bq != B:
            raise ValueError("q batch does not match k")
        qs = (q.stride(0), q.stride(1), q.stride(2))
    if (Hq, Dq) != (H, D):
        raise ValueError(f"q {tuple(q.shape)} does not match k {tuple(k.shape)}")
    if k.dtype not in _cabi.DTYPE_CODE:
        raise TypeError(f"unsupported dtype {k.dtype}")
    p = FlareProblem()
    p.B, p.H, p.N, p.M, p.D = B, H, N, M, D
    p.dtype = _cabi.DTYPE_CODE[k.dtype]
    p.scale = float(scale)
    p.n_splits = int(n_splits)
    p.dropout_p = float(dropout_p)
    p.dropout_seed = int(dropout_seed) & 0xFFFFFFFFFFFFFFFF
    p.q_stride[:] = qs
    p.k_stride[:] = k.stride()[:3]
    for name, t in (("v_stride", v), ("y_stride", y), ("dy_stride", dy), ("dk_stride", dk), ("dv_stride", dv)):
        if t is not None:
            getattr(p, name)[:] = t.stride()[:3]
    return p


def _seed64(seed) -> int:
    """Any integer seed as the operator's signed 64 bits (the kernels see it modulo 2^64)."""
    return ((int(seed) + (1 << 63)) & 0xFFFFFFFFFFFFFFFF) - (1 << 63)


def mixer_forward(q, k, v, scale=1.0, key_mask=None, dropout_p=0.0, dropout_seed=0):
    """y, z32[B,H,M,D], lse_m[B,H,M], lse_n[B,H,N] via flare_mixer_fwd; not recorded by autograd."""
    _need_cuda(q, k, v)
    if not (q.dtype == k.dtype == v.dtype):
        raise TypeError("q, k, v must share a dtype")
    with torch.no_grad():
        return ops.mixer_fwd(q, k, v, float(scale), key_mask, float(dropout_p), _seed64(dropout_seed))


def mixer_backward(q, k, v, dy, y, z32, lse_m, lse_n, scale=1.0, key_mask=None, dropout_p=0.0, dropout_seed=0):
    """dq (fp32, [H,M,D] or [B,H,M,D]), dk, dv via flare_mixer_bwd."""
    _need_cuda(q, k, v, dy, y)
    with torch.no_grad():
        return ops.mixer_bwd(q, k, v, dy, y, z32, lse_m, lse_n, float(scale), key_mask, float(dropout_p), _seed64(dropout_seed))


def gather_forward(q, k, v, scale=1.0, key_mask=None):
    """z (input dtype), z32, lse_m[B,H,M] via flare_gather_partial + flare_combine; not recorded by autograd."""
    _need_cuda(q, k, v)
    with torch.no_grad():
        return ops.gather_fwd(q, k, v, float(scale), key_mask)


def gather_backward(q, k, v, dz, z32, lse_m, scale=1.0, key_mask=None):
    """dq (fp32), dk, dv of the gather alone (term 1 of the backward)."""
    with torch.no_grad():
        return ops.gather_bwd(q, k, v, dz, z32, lse_m, float(scale), key_mask)


def scatter_forward(q, k, z, scale=1.0, key_mask=None):
    """y, lse_n[B,H,N] via flare_scatter; not recorded by autograd."""
    _need_cuda(q, k, z)
    with torch.no_grad():
        return ops.scatter_fwd(q, k, z, float(scale), key_mask)


def scatter_backward(q, k, z, dy, y, lse_n, scale=1.0, key_mask=None):
    """dq (fp32), dk, dz (fp32) of the scatter alone (term 2 of the backward)."""
    with torch.no_grad():
        return ops.scatter_bwd(q, k, z, dy, y, lse_n, float(scale), key_mask)


# ------------------------------------------------------------------------------------
# torch operators: opaque to torch.compile (the fake kernels below give the shapes), differentiable,
# autocast-aware.  The reference runs this path under torch.compile and torch.autocast
# (mlutils/trainer.py:135-137, 185; ablation/time_memory_bwd.py:460-470).  Their CUDA and autograd
# kernels are native code (csrc/binding/flare_torch.cpp).
# ------------------------------------------------------------------------------------
def _like_tokens(k):
    """What the kernels return for a [B,H,N,D] result: k's strides when those are addressable, else dense."""
    e = k.element_size()
    if k.stride(-1) == 1 and all((s * e) % 16 == 0 for s in k.stride()[:-1]):
        out = torch.empty_like(k)
        if out.stride(-1) == 1:
            return out
    return torch.empty(k.shape, dtype=k.dtype, device=k.device)


def _f32(shape, like):
    return torch.empty(shape, dtype=torch.float32, device=like.device)


@torch.library.register_fake("flare_b200::mixer_fwd")
def _(q, k, v, scale, key_mask, dropout_p, dropout_seed):
    B, H, N, D = k.shape
    M = q.shape[-2]
    return _like_tokens(k), _f32((B, H, M, D), k), _f32((B, H, M), k), _f32((B, H, N), k)


@torch.library.register_fake("flare_b200::mixer_bwd")
def _(q, k, v, dy, y, z32, lse_m, lse_n, scale, key_mask, dropout_p, dropout_seed):
    return _f32(q.shape, q), _like_tokens(k), _like_tokens(v)


@torch.library.register_fake("flare_b200::gather_fwd")
def _(q, k, v, scale, key_mask):
    B, H, N, D = k.shape
    M = q.shape[-2]
    return torch.empty(B, H, M, D, dtype=k.dtype, device=k.device), _f32((B, H, M, D), k), _f32((B, H, M), k)


@torch.library.register_fake("flare_b200::gather_bwd")
def _(q, k, v, dz, z32, lse_m, scale, key_mask):
    return _f32(q.shape, q), torch.empty(k.shape, dtype=k.dtype, device=k.device), torch.empty(v.shape, dtype=v.dtype, device=v.device)


@torch.library.register_fake("flare_b200::scatter_fwd")
def _(q, k, z, scale, key_mask):
    B, H, N, D = k.shape
    return _like_tokens(k), _f32((B, H, N), k)


@torch.library.register_fake("flare_b200::scatter_bwd")
def _(q, k, z, dy, y, lse_n, scale, key_mask):
    return _f32(q.shape, q), torch.empty(k.shape, dtype=k.dtype, device=k.device), _f32(z.shape, z)


# ------------------------------------------------------------------------------------
# the public functions
# ------------------------------------------------------------------------------------
def _fold_q(q):
    # an expand()-ed q (stride 0 over the batch, pdebench/models/flare.py:136) is the shared-latent case
    if q.dim() == 4 and q.stride(0) == 0:
        return q[0]
    return q


def _autocast(*ts):
    """What SDPA does under torch.autocast: floating-point CUDA inputs are cast to the autocast dtype, so that
    fp32 latent parameters meet half-precision projections (mlutils/trainer.py:135-137 runs every step so)."""
    if torch.is_autocast_enabled("cuda"):
        dt = torch.get_autocast_dtype("cuda")
        return tuple(t.to(dt) if t is not None and t.is_cuda and t.is_floating_point() else t for t in ts)
    return ts


def _same_dtype(q, k, v):
    if not (q.dtype == k.dtype == v.dtype):
        raise TypeError(f"q, k, v must share a dtype outside torch.autocast; got {q.dtype}, {k.dtype}, {v.dtype}")


_dropout_calls = 0


def next_dropout_seed() -> int:
    """A new 64-bit seed per call, reproducible from torch.manual_seed and the order of the calls."""
    global _dropout_calls
    _dropout_calls += 1
    x = (torch.initial_seed() * 0x9E3779B97F4A7C15 + _dropout_calls * 0xD1B54A32D192ED03) & 0xFFFFFFFFFFFFFFFF
    x ^= x >> 31
    x = (x * 0xBF58476D1CE4E5B9) & 0xFFFFFFFFFFFFFFFF
    x ^= x >> 29
    return x & 0x7FFFFFFFFFFFFFFF


def flare_multihead_mixer(q, k, v, scale: float = 1.0, key_mask: Optional[torch.Tensor] = None,
                          dropout_p: float = 0.0, dropout_seed: Optional[int] = None):
    """y[B,H,N,D] = SDPA(k, q, SDPA(q, k, v, scale), scale)   (README.md:37-53 of the reference).

    q: [H,M,D] (or [B,H,M,D]); k, v: [B,H,N,D], any strides with unit stride on D.
    key_mask: optional bool [B,N], True = token takes part (lra/models/backends.py:615-622);
    masked tokens are ignored by the gather and their output rows are zero.
    dropout_p: attention dropout of both SDPA calls (lra/models/backends.py:604-606): each softmax weight is
    dropped with this probability after normalisation and the rest scaled by 1/(1-p), independently in the
    gather and in the scatter; the masks come from a counter hash of torch's seed (``torch.manual_seed``) and
    the number of dropout calls made so far, not from torch's Philox stream (equal in distribution, not bit
    for bit).  ``dropout_seed`` fixes the masks explicitly.  16-bit dtypes with D in {16, 32} only.
    Works under torch.autocast (inputs are cast to the autocast dtype, as SDPA does) and inside
    torch.compile (registered operators ``flare_b200::mixer_fwd`` / ``mixer_bwd``).
    """
    if q.dim() == 4:
        q = _fold_q(q)
    if torch.is_autocast_enabled("cuda"):
        # what SDPA does: 16-bit k and v, and the latents rounded to them (inside the operator when they are fp32)
        dt = torch.get_autocast_dtype("cuda")
        if k.dtype != dt or v.dtype != dt:
            k, v = _autocast(k, v)
        if q.dtype != dt and (q.dtype != torch.float32 or torch.compiler.is_compiling()):
            q, = _autocast(q)
        if k.dtype != v.dtype or (q.dtype != k.dtype and (q.dtype != torch.float32 or k.dtype != dt)):
            _same_dtype(q, k, v)
    elif not q.dtype == k.dtype == v.dtype:
        _same_dtype(q, k, v)
    seed = 0
    if dropout_p != 0.0:
        if not 0.0 <= dropout_p < 1.0:
            raise ValueError(f"dropout_p must be in [0, 1), got {dropout_p}")
        if k.dtype == torch.float32:
            raise NotImplementedError("attention dropout runs on the tensor-core kernels: bf16 or fp16 inputs (or autocast)")
        seed = next_dropout_seed() if dropout_seed is None else int(dropout_seed)
    if torch.compiler.is_compiling():
        _need_cuda(q, k, v)
        return ops.mixer_fwd(q, k, v, float(scale), key_mask, float(dropout_p), seed)[0]
    return native.mixer(q, k, v, float(scale), key_mask, float(dropout_p), seed)


def flare_gather(q, k, v, scale: float = 1.0, key_mask=None):
    """(z[B,H,M,D], lse[B,H,M]): the first SDPA call, z = softmax_N(scale q k^T) v."""
    _need_cuda(q, k, v)
    q, k, v = _autocast(_fold_q(q), k, v)
    _same_dtype(q, k, v)
    z, _z32, lse_m = ops.gather_fwd(q, k, v, float(scale), key_mask)
    return z, lse_m.detach()


def flare_scatter(q, k, z, scale: float = 1.0, key_mask=None):
    """y[B,H,N,D]: the second SDPA call, y = softmax_M(scale k q^T) z."""
    _need_cuda(q, k, z)
    q, k, z = _autocast(_fold_q(q), k, z)
    return ops.scatter_fwd(q, k, z, float(scale), key_mask)[0]
