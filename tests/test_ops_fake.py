"""The registered torch operators on fake tensors: the shapes, strides and dtypes torch.compile will see,
without a GPU.  (The autograd engine itself needs a live device for CUDA tensors, so the backward operators
are called directly here; differentiation end to end is covered by the GPU tests.)"""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.utils._python_dispatch import TorchDispatchMode

import flare_b200 as fb

ops = torch.ops.flare_b200


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_mixer_operator_shapes_on_fake_tensors(dtype):
    B, H, N, M, D = 2, 4, 300, 32, 16
    with FakeTensorMode():
        x = torch.empty(B, N, H * D, dtype=dtype, device="cuda")
        k = x.view(B, N, H, D).permute(0, 2, 1, 3)           # the 'b n (h d) -> b h n d' view of the reference
        v = (x * 2).view(B, N, H, D).permute(0, 2, 1, 3)
        q = torch.empty(H, M, D, dtype=dtype, device="cuda", requires_grad=True)
        y = fb.flare_multihead_mixer(q.unsqueeze(0).expand(B, -1, -1, -1), k, v, scale=0.5)
        assert y.shape == (B, H, N, D) and y.dtype == dtype and y.requires_grad
        assert y.stride() == k.stride()                      # 'b h n d -> b n (h d)' stays a free view
        y0, z32, lse_m, lse_n = ops.mixer_fwd(q, k, v, 0.5, None, 0.0, 0)
        assert z32.shape == (B, H, M, D) and lse_m.shape == (B, H, M) and lse_n.shape == (B, H, N)
        dq, dk, dv = ops.mixer_bwd(q, k, v, torch.empty_like(y0), y0, z32, lse_m, lse_n, 0.5, None, 0.0, 0)
        assert dq.shape == q.shape and dq.dtype == torch.float32
        assert dk.shape == k.shape and dk.stride() == k.stride() and dv.dtype == dtype


def test_separate_operators_on_fake_tensors():
    B, H, N, M, D = 1, 2, 100, 16, 32
    with FakeTensorMode():
        q = torch.empty(H, M, D, device="cuda", requires_grad=True)
        k = torch.empty(B, H, N, D, device="cuda")
        v = torch.empty(B, H, N, D, device="cuda")
        mask = torch.ones(B, N, dtype=torch.bool, device="cuda")
        z, lse = fb.flare_gather(q, k, v, key_mask=mask)
        assert z.shape == (B, H, M, D) and lse.shape == (B, H, M) and not lse.requires_grad
        y = fb.flare_scatter(q, k, z * 2, key_mask=mask)
        assert y.shape == (B, H, N, D) and y.requires_grad
        dq, dk, dz = ops.scatter_bwd(q, k, z, torch.empty_like(y), y, torch.empty(B, H, N, device="cuda"), 1.0, mask)
        assert dq.shape == q.shape and dk.shape == k.shape and dz.shape == z.shape
        dq, dk, dv = ops.gather_bwd(q, k, v, dz, torch.empty(B, H, M, D, device="cuda"), lse, 1.0, mask)
        assert dq.shape == q.shape and dk.shape == k.shape and dv.shape == v.shape


def test_autocast_casts_the_latents_like_sdpa(monkeypatch):
    B, H, N, M, D = 1, 2, 64, 8, 16
    state = {"on": False}
    # torch.autocast("cuda") switches itself off on a machine without a GPU: stand in for its two queries
    monkeypatch.setattr(torch, "is_autocast_enabled", lambda *a: state["on"])
    monkeypatch.setattr(torch, "get_autocast_dtype", lambda *a: torch.float16)
    with FakeTensorMode():
        q = torch.empty(H, M, D, device="cuda", requires_grad=True)              # fp32 parameter
        k = torch.empty(B, H, N, D, device="cuda", dtype=torch.float16)
        v = torch.empty(B, H, N, D, device="cuda", dtype=torch.float16)
        state["on"] = True
        y = fb.flare_multihead_mixer(q, k, v)
        state["on"] = False
        assert y.dtype == torch.float16 and y.requires_grad
        with pytest.raises(TypeError):
            fb.flare_multihead_mixer(q, k, v)                                    # no autocast: dtypes must agree
        y = fb.flare_multihead_mixer(q.half(), k, v, dropout_p=0.1)               # dropout: a seed is drawn on the host
        assert y.shape == k.shape
        with pytest.raises(NotImplementedError):
            fb.flare_multihead_mixer(q, k.float(), v.float(), dropout_p=0.1)      # fp32 has no dropout kernels
        with pytest.raises(ValueError):
            fb.flare_multihead_mixer(q.half(), k, v, dropout_p=1.0)


@pytest.mark.parametrize("inference,requires_grad", [(True, True), (True, False), (False, False)])
def test_latents_meet_the_operator_in_the_autocast_dtype(monkeypatch, inference, requires_grad):
    """No gradient wanted: the operator's backend kernel gets q rounded, also in inference mode and for inference tensors,
    where the operator's autograd kernel does not run."""
    monkeypatch.setattr(torch, "is_autocast_enabled", lambda *a: True)
    monkeypatch.setattr(torch, "get_autocast_dtype", lambda *a: torch.bfloat16)
    seen = []

    class Record(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            if func is torch.ops.flare_b200.mixer_fwd.default:
                seen.append(tuple(a.dtype for a in args[:3]))
            return func(*args, **(kwargs or {}))

    with FakeTensorMode():
        with torch.inference_mode():
            q, k = (torch.empty(s, device="cuda", dtype=dt) for s, dt in (((2, 8, 16), torch.float32), ((1, 2, 64, 16), torch.bfloat16)))
        if requires_grad:
            q = torch.empty(2, 8, 16, device="cuda", requires_grad=True)
        with torch.inference_mode(inference), Record():
            y = fb.flare_multihead_mixer(q, k, k)
    assert y.dtype == torch.bfloat16 and seen == [(torch.bfloat16,) * 3]


@pytest.mark.parametrize("which,shape", [
    (1, (1, 2, 64, 32)),     # q2 wider than k2: the contraction would read past STATE
    (1, (1, 2, 64, 8)),      # q2 narrower
    (3, (1, 2, 64, 32)),     # k2 wider than q2
    (0, (1, 2, 64, 32)),     # q1 wider than k1
    (2, (1, 2, 64, 32)),     # k1 wider than q1
    (1, (1, 2, 48, 16)),     # fewer tokens than q1
    (4, (1, 2, 48, 16)),     # fewer tokens than k1
    (4, (1, 1, 64, 16)),     # fewer heads
    (3, (2, 64, 16)),        # three dimensions
])
def test_triple_attention_refuses_mismatched_sizes_before_any_launch(which, shape):
    """The refusal comes from the host's size check: nothing is allocated or launched before it."""
    shapes = [(1, 2, 64, 16)] * 5
    shapes[which] = shape
    with FakeTensorMode():
        with pytest.raises(ValueError):
            fb.triple_attention(*(torch.empty(s, dtype=torch.float16, device="cuda") for s in shapes))


@pytest.mark.parametrize("q_dtype,kv_dtype", [(torch.int32, torch.bfloat16), (torch.bool, torch.bfloat16), (torch.int64, torch.float32),
                                             (torch.float32, torch.int32)])
def test_latents_that_autocast_does_not_cast_are_refused(monkeypatch, q_dtype, kv_dtype):
    """Autocast casts floating inputs only: integer latents do not meet 16-bit keys, nor the other way round."""
    monkeypatch.setattr(torch, "is_autocast_enabled", lambda *a: True)
    monkeypatch.setattr(torch, "get_autocast_dtype", lambda *a: torch.bfloat16)
    with FakeTensorMode():
        k = torch.empty(1, 2, 64, 16, device="cuda", dtype=kv_dtype)
        with pytest.raises(TypeError):
            fb.flare_multihead_mixer(torch.empty(2, 8, 16, device="cuda", dtype=q_dtype), k, k)


@pytest.mark.parametrize("seed", [0, -5, 2 ** 63 - 1, 2 ** 63 + 5, 2 ** 64 - 1, 2 ** 64 + 3])
def test_dropout_seed_of_any_size_reaches_the_operator_modulo_2_64(seed):
    got = []

    class Record(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            if func is ops.mixer_fwd.default:
                got.append(args)
            return func(*args, **(kwargs or {}))

    with FakeTensorMode():
        q, k = (torch.empty(s, device="cuda", dtype=torch.bfloat16) for s in ((2, 8, 16), (1, 2, 64, 16)))
        with Record():
            fb.mixer_forward(q, k, k, dropout_p=0.1, dropout_seed=seed)
            fb.flare_multihead_mixer(q, k, k, "0.5")
    assert got[0][6] % 2 ** 64 == seed % 2 ** 64
    assert got[1][3] == 0.5                              # whatever float() takes is a scale


def test_gather_and_scatter_take_forward_mode_inputs():
    """As the mixer: a call that records no backward runs on the values of dual tensors (it makes no tangent)."""
    import torch.autograd.forward_ad as fw
    with FakeTensorMode():
        q, k = torch.empty(2, 8, 16, device="cuda"), torch.empty(1, 2, 64, 16, device="cuda")
        z = torch.empty(1, 2, 8, 16, device="cuda")
        with fw.dual_level():
            d = fw.make_dual(k, torch.ones_like(k))
            assert fb.flare_gather(q, d, k)[0].shape == z.shape
            assert fb.flare_scatter(q, d, z).shape == k.shape
