"""Causal FLARE: prefill over a whole sequence and recurrent decode on a per-(b, h) state.

The reference links this path (README.md:60) without shipping code, a formula or a test vector (its
figs/flare_decoder.py only animates a decoder diagram), so the definition is this library's own choice:
``y_t = softmax_M(S[:, t]) . z_t`` with ``z_t = softmax_{n <= t}(S) v`` and ``S = scale * q k^T`` -- token t
sees the latent summary of tokens 0..t inclusive, the natural reading of "causal" for the gather and the one
under which decoding token by token reproduces the prefill.  The state is one record per latent,
``[B, H, M, D + 2] = (acc[D], m, l)`` in fp32, the same record the non-causal gather writes per token
range; ``causal_state_init`` gives the empty one.  ``flare_causal_mixer`` is the differentiable form for
training (a whole sequence from an empty prefix); prefill with a carried state and decode are forward only.
"""
from __future__ import annotations

import torch

from ._cabi import native

__all__ = ["causal_state_init", "flare_causal_prefill", "flare_causal_decode", "flare_causal_mixer"]


def causal_state_init(B: int, H: int, M: int, D: int, device) -> torch.Tensor:
    """The record of an empty prefix: acc = 0, m = -inf, l = 0."""
    st = torch.zeros(B, H, M, D + 2, dtype=torch.float32, device=device)
    st[..., D] = float("-inf")
    return st


def flare_causal_prefill(q, k, v, scale: float = 1.0, state=None):
    """All tokens of k, v [B,H,N,D] at once.  Returns (y [B,H,N,D], state after the last token)."""
    return native.causal_prefill(q, k, v, float(scale), state)


def flare_causal_decode(q, k, v, state, scale: float = 1.0):
    """The tokens of k, v [B,H,T,D] (T is usually 1) one after the other; `state` is updated in place."""
    return native.causal_decode(q, k, v, state, float(scale))


def flare_causal_mixer(q, k, v, scale: float = 1.0):
    """Causal FLARE over a whole sequence, differentiable in q, k, v: token t sees the latent summary of
    tokens 0..t only.  q [H,M,D] (or [B,H,M,D]), k, v [B,H,N,D]; returns y [B,H,N,D].

    Where a gradient is wanted, bf16 with M <= 128 and D in {32, 64} keeps the states before every 128-token chunk for
    the backward: M (4 D + 8) bytes per chunk and head, next to q, k and v (138 MB at B = 4, H = 16, N = 8192, M = 128,
    D = 64, where k and v are 134 MB).  They are ordinary saved tensors: torch.utils.checkpoint around the call rebuilds
    them, torch.autograd.graph.save_on_cpu moves them away."""
    return native.causal_mixer(q, k, v, float(scale))
