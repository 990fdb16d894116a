"""Causal FLARE on the GPU against the CPU oracle (dense and recurrent forms).

The reference has no code for this path, so the oracle itself is checked for self-consistency
(tests/test_oracle.py); here the CUDA prefill and decode are compared with it.
"""
import math

import pytest
import torch

from oracle import flare_oracle as O

pytestmark = pytest.mark.gpu

TOL = {torch.float32: 2e-5, torch.bfloat16: 2e-2, torch.float16: 5e-3}


def _inputs(B, H, N, M, D, dtype, seed=0):
    q, k, v, _ = O.make_inputs(B, H, N, M, D, dtype=dtype, seed=seed)
    return q, k, v


@pytest.mark.parametrize("B,H,N,M,D,dtype", [
    (1, 2, 64, 32, 32, torch.float32),
    (2, 2, 200, 64, 32, torch.float32),       # ragged: 1.56 chunks, partial sub-chunk
    (1, 2, 384, 128, 64, torch.float32),      # the serving shape's M and D
    (1, 2, 300, 256, 32, torch.bfloat16),
    (2, 3, 257, 128, 64, torch.bfloat16),
    (1, 1, 130, 64, 16, torch.float16),
])
def test_prefill_matches_oracle(cuda_dev, B, H, N, M, D, dtype):
    import flare_b200 as fb
    q, k, v = _inputs(B, H, N, M, D, dtype)
    y_ref, (m_ref, l_ref, a_ref) = O.causal_recurrent(q.double(), k.double(), v.double(), 1.0)
    y, st = fb.flare_causal_prefill(q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev), 1.0)
    assert O.rel_l2(y.double().cpu(), y_ref) <= TOL[dtype]
    # the final record, compared through what it represents: z = acc / l and lse = m + log l
    st = st.double().cpu()
    z = st[..., :D] / st[..., D + 1:D + 2]
    lse = st[..., D] + torch.log(st[..., D + 1])
    assert O.rel_l2(z, a_ref / l_ref[..., None]) <= TOL[dtype]
    assert O.rel_l2(lse, m_ref + torch.log(l_ref)) <= TOL[dtype]


def test_prefill_dense_small(cuda_dev):
    import flare_b200 as fb
    q, k, v = _inputs(1, 2, 40, 16, 16, torch.float32, seed=3)
    y_ref = O.causal_dense(q.double(), k.double(), v.double(), 0.7)
    y, _ = fb.flare_causal_prefill(q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev), 0.7)
    assert O.rel_l2(y.double().cpu(), y_ref) <= 2e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_decode_continues_prefill(cuda_dev, dtype):
    """prefill(first part) then token-by-token decode == prefill(everything)."""
    import flare_b200 as fb
    B, H, N, M, D = 2, 2, 160, 64, 32
    q, k, v = _inputs(B, H, N, M, D, dtype, seed=5)
    qd, kd, vd = q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev)
    y_all, st_all = fb.flare_causal_prefill(qd, kd, vd, 1.0)
    n0 = 100
    y0, st = fb.flare_causal_prefill(qd, kd[:, :, :n0], vd[:, :, :n0], 1.0)
    ys = [y0]
    for t in range(n0, N - 8):
        ys.append(fb.flare_causal_decode(qd, kd[:, :, t:t + 1], vd[:, :, t:t + 1], st, 1.0))
    ys.append(fb.flare_causal_decode(qd, kd[:, :, N - 8:], vd[:, :, N - 8:], st, 1.0))   # several tokens in one call
    y_inc = torch.cat(ys, dim=2)
    y_ref, _ = O.causal_recurrent(q.double(), k.double(), v.double(), 1.0)
    assert O.rel_l2(y_inc.double().cpu(), y_ref) <= TOL[dtype]
    assert O.rel_l2(y_inc.double().cpu(), y_all.double().cpu()) <= TOL[dtype]


def test_decode_from_empty_state(cuda_dev):
    import flare_b200 as fb
    B, H, N, M, D = 1, 2, 24, 32, 32
    q, k, v = _inputs(B, H, N, M, D, torch.float32, seed=7)
    st = fb.causal_state_init(B, H, M, D, cuda_dev)
    y = fb.flare_causal_decode(q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev), st, 1.0)
    y_ref, _ = O.causal_recurrent(q.double(), k.double(), v.double(), 1.0)
    assert O.rel_l2(y.double().cpu(), y_ref) <= 2e-5


def test_prefill_with_prior_state(cuda_dev):
    import flare_b200 as fb
    B, H, N, M, D = 1, 2, 300, 64, 32
    q, k, v = _inputs(B, H, N, M, D, torch.float32, seed=9)
    qd, kd, vd = q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev)
    _, st = fb.flare_causal_prefill(qd, kd[:, :, :128], vd[:, :, :128], 1.0)
    y2, _ = fb.flare_causal_prefill(qd, kd[:, :, 128:], vd[:, :, 128:], 1.0, state=st)
    y_ref, _ = O.causal_recurrent(q.double(), k.double(), v.double(), 1.0)
    assert O.rel_l2(y2.double().cpu(), y_ref[:, :, 128:]) <= 2e-5


def test_unsupported_shape_is_refused(cuda_dev):
    import flare_b200 as fb
    q, k, v = _inputs(1, 1, 16, 520, 64, torch.float32)
    with pytest.raises(Exception):
        fb.flare_causal_prefill(q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev), 1.0)


def test_serving_shape_split_prefill(cuda_dev):
    """B=4, H=16, N=8192, D=64, M=128 bf16 (too large for the CPU oracle): prefilling the prompt in two pieces
    with the carried record, and decoding its last tokens one by one, give what one prefill gives."""
    import flare_b200 as fb
    B, H, N, M, D = 4, 16, 8192, 128, 64
    g = torch.Generator().manual_seed(31)
    q = (torch.randn(H, M, D, generator=g) * D ** -0.25).bfloat16().to(cuda_dev)
    k = (torch.randn(B, H, N, D, generator=g) * D ** -0.25).bfloat16().to(cuda_dev)
    v = torch.randn(B, H, N, D, generator=g).bfloat16().to(cuda_dev)
    y_all, st_all = fb.flare_causal_prefill(q, k, v, 1.0)
    n0 = 5000                                            # not a multiple of the chunk
    y0, st = fb.flare_causal_prefill(q, k[:, :, :n0], v[:, :, :n0], 1.0)
    y1, st = fb.flare_causal_prefill(q, k[:, :, n0:N - 16], v[:, :, n0:N - 16], 1.0, state=st)
    ys = [y0, y1]
    for t in range(N - 16, N):
        ys.append(fb.flare_causal_decode(q, k[:, :, t:t + 1], v[:, :, t:t + 1], st, 1.0))
    y_inc = torch.cat(ys, dim=2)
    err = ((y_inc.float() - y_all.float()).norm() / y_all.float().norm()).item()
    assert err <= 2e-2, err
    z_a = st_all[..., :D] / st_all[..., D + 1:D + 2]
    z_b = st[..., :D] / st[..., D + 1:D + 2]
    assert ((z_a - z_b).norm() / z_a.norm()).item() <= 2e-2


@pytest.mark.parametrize("B,H,N,M,D,shared", [
    (1, 2, 128, 128, 32, False),     # exactly one chunk
    (2, 2, 333, 128, 64, True),      # ragged last chunk, latents shared by the batch
    (1, 3, 700, 64, 64, False),      # fewer latents than tensor-memory lanes
    (2, 1, 130, 96, 32, True),
    (1, 1, 5, 32, 32, False),        # a handful of tokens
])
def test_prefill_tensor_core_walk_shapes(cuda_dev, B, H, N, M, D, shared):
    """bf16 with M <= 128 and D in {32, 64} takes the tensor-core walk; state carried from a prior prefill too."""
    import flare_b200 as fb
    q, k, v = _inputs(B, H, N, M, D, torch.bfloat16, seed=11)          # q: [H, M, D]
    if not shared:                                                      # one latent set per batch element
        q = (torch.randn(B, H, M, D, generator=torch.Generator().manual_seed(12)) * D ** -0.25).bfloat16()
    y_ref, (m_ref, l_ref, a_ref) = O.causal_recurrent(q.double(), k.double(), v.double(), 0.9)
    qd, kd, vd = q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev)
    y, st = fb.flare_causal_prefill(qd, kd, vd, 0.9)
    torch.cuda.synchronize()
    assert fb.device_status() == 0
    assert O.rel_l2(y.double().cpu(), y_ref) <= 2e-2
    if N > 64:                                           # split anywhere: the second call starts from a record
        n0 = N // 3
        y0, st0 = fb.flare_causal_prefill(qd, kd[:, :, :n0].contiguous(), vd[:, :, :n0].contiguous(), 0.9)
        y1, _ = fb.flare_causal_prefill(qd, kd[:, :, n0:].contiguous(), vd[:, :, n0:].contiguous(), 0.9, state=st0)
        assert O.rel_l2(torch.cat([y0, y1], 2).double().cpu(), y_ref) <= 2e-2


def test_prefill_replays_from_a_cuda_graph(cuda_dev):
    """The four chained launches of the tensor-core prefill (records, scan, walk, redo pass) recorded once and replayed
    on new inputs written into the same buffers."""
    import flare_b200 as fb
    B, H, N, M, D = 2, 2, 700, 128, 64
    q, k, v = _inputs(B, H, N, M, D, torch.bfloat16, seed=17)
    q2, k2, v2 = _inputs(B, H, N, M, D, torch.bfloat16, seed=18)
    qd, kd, vd = q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev)
    side = torch.cuda.Stream(device=cuda_dev)
    side.wait_stream(torch.cuda.current_stream(cuda_dev))
    with torch.cuda.stream(side):
        fb.flare_causal_prefill(qd, kd, vd, 1.0)                     # warm-up outside the recording
    torch.cuda.current_stream(cuda_dev).wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y, st = fb.flare_causal_prefill(qd, kd, vd, 1.0)
    for qq, kk, vv in ((q, k, v), (q2, k2, v2)):
        qd.copy_(qq.to(cuda_dev)); kd.copy_(kk.to(cuda_dev)); vd.copy_(vv.to(cuda_dev))
        graph.replay()
        torch.cuda.synchronize()
        y_ref, _ = O.causal_recurrent(qq.double(), kk.double(), vv.double(), 1.0)
        assert O.rel_l2(y.double().cpu(), y_ref) <= 2e-2
    assert fb.device_status() == 0


def test_prefill_tensor_core_walk_hands_wide_chunks_to_the_fp32_walk(cuda_dev):
    """Scores that climb by hundreds of octaves inside one chunk: the tensor-core walk keeps one reference
    maximum per chunk, flags such chunks, and the fp32 walk with a running maximum redoes them."""
    import flare_b200 as fb
    B, H, N, M, D = 1, 2, 384, 64, 32
    q, k, v = _inputs(B, H, N, M, D, torch.bfloat16, seed=13)
    ramp = torch.ones(N)
    ramp[128:256] = torch.linspace(1.0, 60.0, 128)       # the middle chunk only
    k = (k.float() * ramp[None, None, :, None]).bfloat16()
    y_ref, _ = O.causal_recurrent(q.double(), k.double(), v.double(), 1.0)
    y, _ = fb.flare_causal_prefill(q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev), 1.0)
    torch.cuda.synchronize()
    assert fb.device_status() == 0
    assert torch.isfinite(y.float()).all()
    assert O.rel_l2(y.double().cpu(), y_ref) <= 2e-2


# ---------------------------------------------------------------------------------------------------------
# backward (flare_causal_mixer): against autograd through the dense definition and the chunked restatement
# ---------------------------------------------------------------------------------------------------------
def _fb():
    import flare_b200 as fb
    return fb


def _bwd_case(fb, dev, B, H, N, M, D, dtype, scale, seed):
    q, k, v, dy = O.make_inputs(B, H, N, M, D, dtype=dtype, seed=seed)
    qd, kd, vd = (t.to(dev).requires_grad_(True) for t in (q, k, v))
    y = fb.flare_causal_mixer(qd, kd, vd, scale)
    y.backward(dy.to(dev))
    torch.cuda.synchronize()
    assert fb.device_status() == 0
    return (q, k, v, dy), (y.detach().cpu(), qd.grad.cpu(), kd.grad.cpu(), vd.grad.cpu())


@pytest.mark.parametrize("B,H,N,M,D", [(1, 2, 96, 16, 16), (2, 2, 300, 32, 32), (1, 1, 257, 64, 64), (1, 2, 129, 128, 64)])
def test_backward_matches_autograd_of_the_dense_definition(cuda_dev, B, H, N, M, D):
    """fp32 kernel against fp64 autograd through causal_dense: ragged ends (N not a multiple of 32 or 128),
    one to three chunks, every supported head dim."""
    fb = _fb()
    (q, k, v, dy), (y, dq, dk, dv) = _bwd_case(fb, cuda_dev, B, H, N, M, D, torch.float32, 0.8, seed=21)
    qf, kf, vf, dyf = (t.double() for t in (q, k, v, dy))
    dq_ref, dk_ref, dv_ref = O.causal_bwd_autograd(qf, kf, vf, dyf, 0.8)
    assert O.rel_l2(y.double(), O.causal_dense(qf, kf, vf, 0.8)) <= 1e-5
    assert O.rel_l2(dq.double(), dq_ref) <= 1e-4
    assert O.rel_l2(dk.double(), dk_ref) <= 1e-4
    assert O.rel_l2(dv.double(), dv_ref) <= 1e-4


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.bfloat16, 3e-2), (torch.float16, 5e-3)])
def test_backward_long_sequence_against_the_chunked_restatement(cuda_dev, dtype, tol):
    """N = 2000 (16 chunks, ragged last one), latents shared by two batch entries: the carried suffix state
    crosses many chunk boundaries.  The yardstick is the oracle's reverse chunk scan in fp64 on the same
    rounded inputs (itself pinned to autograd on small cases in the CPU suite)."""
    fb = _fb()
    B, H, N, M, D = 2, 2, 2000, 32, 32
    (q, k, v, dy), (y, dq, dk, dv) = _bwd_case(fb, cuda_dev, B, H, N, M, D, dtype, 1.0, seed=22)
    qf, kf, vf, dyf = (t.double() for t in (q, k, v, dy))
    dq_ref, dk_ref, dv_ref = O.causal_bwd_chunked(qf, kf, vf, dyf, 1.0, chunk=64)
    assert O.rel_l2(dq.double(), dq_ref) <= tol
    assert O.rel_l2(dk.double(), dk_ref) <= tol
    assert O.rel_l2(dv.double(), dv_ref) <= tol


@pytest.mark.parametrize("B,H,N,M,D", [
    (1, 2, 128, 128, 64),      # one full chunk: no state handed on
    (2, 3, 333, 128, 64),      # ragged last chunk, latents shared by the batch
    (1, 1, 129, 64, 64),       # a last chunk of one token, fewer latents than rows
    (1, 2, 5, 32, 32),
    (2, 1, 1000, 96, 32),      # a latent count that is no multiple of 64
    (1, 64, 4800, 128, 32),    # 2432 chunks, one to a unit: every CTA takes sixteen or seventeen of them
])
def test_backward_on_tensor_cores(cuda_dev, B, H, N, M, D):
    """bf16 with M <= 128 and D in {32, 64}: one chunk per CTA, the suffix state handed from chunk to chunk.
    Tolerance: the results are rounded to bf16 (1.7e-3 in the 2-norm) and every operand carries a remainder term;
    three times that, since the shortest cases average over a few hundred values only."""
    fb = _fb()
    (q, k, v, dy), (y, dq, dk, dv) = _bwd_case(fb, cuda_dev, B, H, N, M, D, torch.bfloat16, 1.0, seed=N + M)
    ref = O.causal_bwd_chunked(*(t.double() for t in (q, k, v, dy)), 1.0, chunk=128)
    for got, want in zip((dq, dk, dv), ref):
        assert O.rel_l2(got.double(), want) <= 5e-3


@pytest.mark.parametrize("N,M,D", [(512, 128, 64), (700, 64, 32), (385, 100, 64)])
def test_backward_error_is_that_of_rounding_the_results(cuda_dev, N, M, D):
    """bf16 results carry 1.67e-3 of rounding (a uniform error of up to 2^-9 of each value); every operand of the
    tensor-core products has two terms, so nothing near a second rounding (together 2.4e-3) may show."""
    fb = _fb()
    q, k, v, dy = O.make_inputs(1, 4, N, M, D, dtype=torch.bfloat16, seed=N + M)
    qd, kd, vd = (t.to(cuda_dev).requires_grad_(True) for t in (q, k, v))
    fb.flare_causal_mixer(qd, kd, vd, 1.0).backward(dy.to(cuda_dev))
    ref = O.causal_bwd_chunked(q.double(), k.double(), v.double(), dy.double(), 1.0, chunk=128)
    for n, t, r in zip("qkv", (qd, kd, vd), ref):
        assert O.rel_l2(t.grad.double().cpu(), r) < 1.85e-3, n


def _too_wide(q, k, margin=5.0):
    """Whether a head leaves the range of the tensor-core backward in some 128-token chunk: in octaves, a latent's maximum
    climbing by more than 64 after the chunk's first token, or a row or column maximum more than 50 from that token's
    column maximum.  A head within `margin` of a limit is neither."""
    S, top, m0 = (q @ k.t()) / math.log(2.0), -math.inf, torch.full((q.shape[0],), -math.inf, dtype=q.dtype)
    for c in range(0, k.shape[0], 128):
        s = S[:, c:c + 128]
        mu, first, cm = torch.maximum(m0, s.amax(1)), torch.maximum(m0, s[:, 0]), s.amax(0)
        top = max(top, ((mu - first).max() - 64).item(), ((mu - cm[0]).abs().max() - 50).item(), ((cm - cm[0]).abs().max() - 50).item())
        m0 = mu
    assert abs(top) > margin
    return top > 0


def test_backward_hands_wide_heads_to_the_fp32_kernel(cuda_dev):
    """Scores that climb past 64 octaves inside a chunk in one of three heads: that head is redone by the fp32
    kernel (finite, same tolerance), the others stay as they are."""
    fb = _fb()
    B, H, N, M, D = 1, 3, 300, 64, 32
    q, k, v, dy = O.make_inputs(B, H, N, M, D, dtype=torch.bfloat16, seed=29)
    k = k.clone()
    k[:, 1, 128:256] = (k[:, 1, 128:256].float() * torch.linspace(0.1, 40.0, 128).view(1, 128, 1)).bfloat16()
    assert [_too_wide(q[h].double(), k[0, h].double()) for h in range(H)] == [False, True, False]
    qd, kd, vd = (t.to(cuda_dev).requires_grad_(True) for t in (q, k, v))
    y = fb.flare_causal_mixer(qd, kd, vd, 1.0)
    y.backward(dy.to(cuda_dev))
    assert fb.device_status() == 0
    ref = O.causal_bwd_chunked(*(t.double() for t in (q, k, v, dy)), 1.0, chunk=32)
    for got, want in zip((qd.grad, kd.grad, vd.grad), ref):
        assert torch.isfinite(got).all()
        for h in range(H):
            g, r = (got[h], want[h]) if got.dim() == 3 else (got[:, h], want[:, h])
            assert O.rel_l2(g.double().cpu(), r) <= 5e-3, h


def test_c_backward_takes_any_float_pointer_for_the_latent_gradient(cuda_dev):
    """flare_causal_bwd with dq32 at 4 bytes past a 16-byte boundary: the fp32 kernel takes it.  Both forms start from
    16-bit records (below 1e-3 of the fp64 gradient), so they agree to twice that."""
    import ctypes as C
    fb = _fb()
    from flare_b200 import _cabi
    from flare_b200.mixer import make_problem
    B, H, N, M, D = 1, 2, 300, 64, 32
    q, k, v, dy = (t.to(cuda_dev) for t in O.make_inputs(B, H, N, M, D, dtype=torch.bfloat16, seed=35))
    got = []
    for off in (0, 1):
        dk, dv, buf = torch.empty_like(k), torch.empty_like(v), torch.zeros(B * H * M * D + 4, device=cuda_dev)
        dq = buf[off:off + B * H * M * D]
        p = make_problem(q, k, 1.0, v=v, dy=dy, dk=dk, dv=dv)
        ws = torch.empty(_cabi.lib.flare_causal_bwd_workspace_bytes(C.byref(p)), dtype=torch.uint8, device=cuda_dev)
        _cabi.check(_cabi.lib.flare_causal_bwd(C.byref(p), *(_cabi.ptr(t) for t in (q, k, v, dy, dq, dk, dv, ws)), _cabi.stream_of(q)), "bwd")
        got.append(dq.clone())
    assert fb.device_status() == 0
    assert O.rel_l2(got[1], got[0]) <= 2e-3


@pytest.mark.parametrize("how", ["checkpoint", "save_on_cpu"])
def test_kept_states_can_be_rebuilt_or_moved_away(cuda_dev, how):
    """The chunk-start states of the training forward are ordinary saved tensors."""
    from torch.utils.checkpoint import checkpoint
    fb = _fb()
    q, k, v, dy = (t.to(cuda_dev) for t in O.make_inputs(1, 4, 1000, 128, 64, dtype=torch.bfloat16, seed=36))
    x = [t.requires_grad_(True) for t in (q, k, v)]
    want = torch.autograd.grad(fb.flare_causal_mixer(*x, 1.0), x, dy)
    if how == "checkpoint":
        y = checkpoint(fb.flare_causal_mixer, *x, 1.0, use_reentrant=False)
    else:
        with torch.autograd.graph.save_on_cpu():
            y = fb.flare_causal_mixer(*x, 1.0)
    for a, b in zip(torch.autograd.grad(y, x, dy), want):
        assert torch.equal(a, b)


def test_mixer_without_gradients_is_the_plain_prefill(cuda_dev):
    """No gradient wanted: the kernels of the prefill, to the bit (the training forward keeps its chunk prefixes in two terms)."""
    fb = _fb()
    q, k, v, dy = (t.to(cuda_dev) for t in O.make_inputs(2, 4, 2000, 128, 64, dtype=torch.bfloat16, seed=24))
    want, _ = fb.flare_causal_prefill(q, k, v, 1.0)
    assert torch.equal(fb.flare_causal_mixer(q, k, v, 1.0), want)
    q.requires_grad_(True)
    with torch.no_grad():
        assert torch.equal(fb.flare_causal_mixer(q, k, v, 1.0), want)
    with torch.inference_mode():
        assert torch.equal(fb.flare_causal_mixer(q, k, v, 1.0), want)
    y = fb.flare_causal_mixer(q, k, v, 1.0)                  # a gradient for q alone: the training forward
    dq, = torch.autograd.grad(y, q, dy)
    ref, _, _ = O.causal_bwd_chunked(*(t.detach().double().cpu() for t in (q, k, v, dy)), 1.0, chunk=128)
    assert O.rel_l2(dq.double().cpu(), ref) <= 5e-3


def test_backward_with_growing_logits(cuda_dev):
    """Keys whose norm grows along the sequence: the running maxima rise by tens of units from chunk to
    chunk, so the carried suffix state is rescaled by tiny factors and early tokens' weights underflow
    relative to late maxima -- finite results that match the fp64 restatement."""
    fb = _fb()
    B, H, N, M, D = 1, 2, 640, 32, 32
    q, k, v, dy = O.make_inputs(B, H, N, M, D, dtype=torch.float32, seed=23)
    k = k * torch.linspace(0.5, 6.0, N).view(1, 1, N, 1)
    qd, kd, vd = (t.to(cuda_dev).requires_grad_(True) for t in (q, k, v))
    y = fb.flare_causal_mixer(qd, kd, vd, 1.0)
    y.backward(dy.to(cuda_dev))
    qf, kf, vf, dyf = (t.double() for t in (q, k, v, dy))
    dq_ref, dk_ref, dv_ref = O.causal_bwd_chunked(qf, kf, vf, dyf, 1.0, chunk=32)
    for got, ref in ((qd.grad, dq_ref), (kd.grad, dk_ref), (vd.grad, dv_ref)):
        assert torch.isfinite(got).all()
        assert O.rel_l2(got.cpu().double(), ref) <= 2e-4


def test_backward_refuses_what_it_cannot_hold(cuda_dev):
    fb = _fb()
    q, k, v, dy = O.make_inputs(1, 1, 64, 64, 128, dtype=torch.float32, seed=1)   # forward: fine; backward: D = 128
    qd, kd, vd = (t.to(cuda_dev).requires_grad_(True) for t in (q, k, v))
    y = fb.flare_causal_mixer(qd, kd, vd, 1.0)
    with pytest.raises(RuntimeError, match="causal_bwd"):
        y.backward(dy.to(cuda_dev))


# ---------------------------------------------------------------------------------------------------------
# the call-site variants of the reference's FLARE modules on the serving path
# ---------------------------------------------------------------------------------------------------------
def test_decode_with_shared_latents_and_normalised_q_k(cuda_dev):
    """`shared_latents` (one latent set expand()-ed over the heads: stride 0) and `qk_norm` (q, k normalised
    by the caller before the mixer; pdebench/models/flare.py:130-132) on prefill + decode: the broadcast view is
    accepted as it is, and what comes out equals the oracle on the materialised, normalised tensors."""
    import flare_b200 as fb
    import torch.nn.functional as F
    B, H, N, M, D = 2, 4, 150, 32, 32
    g = torch.Generator().manual_seed(31)
    q1 = torch.randn(1, M, D, generator=g)
    k = torch.randn(B, H, N, D, generator=g)
    v = torch.randn(B, H, N, D, generator=g)
    qn = F.normalize(q1, dim=-1).expand(H, M, D)            # stride 0 over the heads
    kn = F.normalize(k, dim=-1)
    assert qn.stride(0) == 0
    scale = 4.0                                             # unit vectors: a sharper softmax than scale 1
    qd, kd, vd = qn.to(cuda_dev), kn.to(cuda_dev), v.to(cuda_dev)
    qd = qd[:1].expand(H, M, D)                             # (.to() materialises; make the device view broadcast again)
    n0 = 128
    y0, st = fb.flare_causal_prefill(qd, kd[:, :, :n0], vd[:, :, :n0], scale)
    ys = [y0] + [fb.flare_causal_decode(qd, kd[:, :, t:t + 1], vd[:, :, t:t + 1], st, scale) for t in range(n0, N)]
    y = torch.cat(ys, dim=2)
    y_ref, _ = O.causal_recurrent(qn.contiguous().double(), kn.double(), v.double(), scale)
    assert O.rel_l2(y.double().cpu(), y_ref) <= 2e-5


def test_training_step_with_shared_latents(cuda_dev):
    """flare_causal_mixer with the latents expand()-ed over the heads: autograd folds the per-head gradients
    back onto the single latent set, equal to autograd through the dense definition."""
    import flare_b200 as fb
    B, H, N, M, D = 1, 3, 100, 16, 16
    g = torch.Generator().manual_seed(32)
    q1 = (torch.randn(1, M, D, generator=g) * 0.5)
    k = torch.randn(B, H, N, D, generator=g) * 0.5
    v = torch.randn(B, H, N, D, generator=g)
    dy = torch.randn(B, H, N, D, generator=g)
    qd = q1.to(cuda_dev).requires_grad_(True)
    kd, vd = k.to(cuda_dev).requires_grad_(True), v.to(cuda_dev).requires_grad_(True)
    fb.flare_causal_mixer(qd.expand(H, M, D), kd, vd, 1.0).backward(dy.to(cuda_dev))
    qr = q1.double().requires_grad_(True)
    kr, vr = k.double().requires_grad_(True), v.double().requires_grad_(True)
    O.causal_dense(qr.expand(H, M, D), kr, vr, 1.0).backward(dy.double())
    assert O.rel_l2(qd.grad.double().cpu(), qr.grad) <= 1e-4
    assert O.rel_l2(kd.grad.double().cpu(), kr.grad) <= 1e-4
    assert O.rel_l2(vd.grad.double().cpu(), vr.grad) <= 1e-4


@pytest.mark.parametrize("dtype,M,tol", [(torch.bfloat16, 32, 5e-3), (torch.bfloat16, 160, 3e-2), (torch.float32, 32, 1e-4)])
def test_gradient_of_batch_expanded_latents(cuda_dev, dtype, M, tol):
    """One latent set expand()-ed over the batch and differentiated itself: every batch entry has its own gradient (on
    the tensor-core shapes and on the others), and the set below it gets their sum."""
    import flare_b200 as fb
    B, H, N, D = 3, 2, 300, 32
    q, k, v, dy = O.make_inputs(B, H, N, M, D, dtype=dtype, seed=33)
    q1 = q.to(cuda_dev).requires_grad_(True)
    qe = q1.unsqueeze(0).expand(B, -1, -1, -1)
    kd, vd = k.to(cuda_dev).requires_grad_(True), v.to(cuda_dev).requires_grad_(True)
    y = fb.flare_causal_mixer(qe, kd, vd, 1.0)
    got = torch.autograd.grad(y, (qe, q1, kd, vd), dy.to(cuda_dev))
    qf = q.double().unsqueeze(0).repeat(B, 1, 1, 1)
    dq, dk, dv = O.causal_bwd_chunked(qf, *(t.double() for t in (k, v, dy)), 1.0, chunk=64)
    assert got[0].shape == dq.shape
    for b in range(B):
        assert O.rel_l2(got[0][b].double().cpu(), dq[b]) <= tol
    for g, r in zip(got[1:], (dq.sum(0), dk, dv)):
        assert O.rel_l2(g.double().cpu(), r) <= tol


def test_decode_step_replays_from_a_cuda_graph(cuda_dev):
    """The serving loop: one decode step recorded in a CUDA graph over static k_t, v_t, y_t buffers and the
    state record, replayed once per token (the state lives in one fp32 tensor updated in place, so the
    recorded launch needs nothing new per step).  Equals the prefill over the same tokens."""
    import flare_b200 as fb
    B, H, N, M, D = 2, 4, 96, 64, 32
    q, k, v = _inputs(B, H, N, M, D, torch.bfloat16, seed=41)
    qd, kd, vd = q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev)
    n0 = 32
    _, st = fb.flare_causal_prefill(qd, kd[:, :, :n0], vd[:, :, :n0], 1.0)
    k_t = torch.empty(B, H, 1, D, dtype=torch.bfloat16, device=cuda_dev)
    v_t = torch.empty_like(k_t)
    k_t.copy_(kd[:, :, n0:n0 + 1]); v_t.copy_(vd[:, :, n0:n0 + 1])
    side = torch.cuda.Stream(device=cuda_dev)
    side.wait_stream(torch.cuda.current_stream(cuda_dev))
    st_warm = st.clone()
    with torch.cuda.stream(side):
        fb.flare_causal_decode(qd, k_t, v_t, st_warm, 1.0)          # warm-up outside the recording
    torch.cuda.current_stream(cuda_dev).wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y_t = fb.flare_causal_decode(qd, k_t, v_t, st, 1.0)
    ys = []
    for t in range(n0, N):
        k_t.copy_(kd[:, :, t:t + 1]); v_t.copy_(vd[:, :, t:t + 1])
        graph.replay()
        ys.append(y_t.clone())
    torch.cuda.synchronize()
    y_all, st_all = fb.flare_causal_prefill(qd, kd, vd, 1.0)
    assert O.rel_l2(torch.cat(ys, dim=2).float().cpu(), y_all[:, :, n0:].float().cpu()) <= 2e-2
    z = lambda s: (s[..., :D] / s[..., D + 1:D + 2]).cpu()
    assert O.rel_l2(z(st), z(st_all)) <= 2e-2          # (the prefill state comes from the bf16 tensor-core gather)
    assert fb.device_status() == 0
