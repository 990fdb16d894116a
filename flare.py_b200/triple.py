"""Triple attention and causal linear attention over the C ABI.

``triple_attention(q1, q2, k1, k2, v)`` has the meaning of ``TripleAttentionFunction`` in the reference
(lra/models/triton/triple.py:27-290; einsum form :846-860): it returns ``(STATE, O)`` with
``STATE[b,h,i,j,k] = (1/N) sum_n K1[n,i] V[n,j] K2[n,k]`` (fp32) and
``O[n,j] = sum_{i,k} Q1[n,i] STATE[i,j,k] Q2[n,k]``, and is differentiable (backward formulas :887-931).
``causal_linear(q, k, v)`` is ``CausalLinear`` (lra/models/triton/causal_linear.py:23-145, reference
:317-336): ``Y_t = Q_t sum_{n<=t} K_n^T V_n / N``, forward only as there.
"""
from __future__ import annotations

from ._cabi import native

__all__ = ["triple_attention", "causal_linear"]


def triple_attention(q1, q2, k1, k2, v):
    """(STATE [B,H,Dq,Dv,Dq] fp32, O [B,H,N,Dv]); q1, q2, k1, k2: [B,H,N,Dq], v: [B,H,N,Dv]."""
    return native.triple(q1, q2, k1, k2, v)


def causal_linear(q, k, v):
    """Y [B,H,N,Dv] = Q_t . sum_{n<=t} K_n^T V_n / N; q, k: [B,H,N,Dk], v: [B,H,N,Dv]."""
    return native.causal_linear(q, k, v)
