"""fp32 inputs (the reference's CPU-runnable correctness configuration): |err| <= 1e-4 on O, lse, dQ, dK, dV
against the fp32 CPU oracle, through the Python entry points."""
import math

import pytest
import torch

import _parity
from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu
SCALE = 1.0 / math.sqrt(128.0)


def run(device, B, Hq, Hkv, Sq, Skv, seed, kv_valid=None):
    import lv_xattn_b200 as lvx
    from lv_xattn_b200 import _lib
    q, k, v, do = orc.make_inputs(B, Hq, Hkv, Sq, Skv, 128, seed, torch.float32)
    ref = orc.attention_fwd_bwd(q, k, v, do, SCALE, kv_valid)
    qd, kd, vd, dod = (t.to(device) for t in (q, k, v, do))
    _, _, _, o, L = lvx._attn_forward(qd, kd, vd, False, SCALE, None, kv_valid_len=kv_valid)
    dq, dk, dv = lvx._attn_backward(dod, qd, kd, vd, o, L, False, SCALE, None, "flash", kv_valid_len=kv_valid)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    assert o.dtype == torch.float32 and dq.dtype == torch.float32
    got = (o.cpu(), L.cpu().view(B, Hq, Sq), dq.cpu(), dk.cpu(), dv.cpu())
    return got, ref


def check(got, ref, tol=1e-4):
    _parity.assert_lse_close(got[1], ref[1], "fp32", tol)
    for name, g, r in zip(("o", "lse", "dq", "dk", "dv"), got, ref):
        if name != "lse":
            _parity.assert_fp32(g, r, name, "fp32")


def test_config1_shape(cuda_device):
    # B=1, 32 query heads, 8 KV heads, 512 queries, 8192 keys, fp32, no mask, scale 1/sqrt(128)
    check(*run(cuda_device, 1, 32, 8, 512, 8192, 1))


@pytest.mark.parametrize("shape", [(1, 1, 1, 64, 64), (2, 4, 2, 40, 200), (1, 8, 2, 96, 1000)])
def test_small_and_ragged(cuda_device, shape):
    check(*run(cuda_device, *shape, 2))


def test_key_padding(cuda_device):
    check(*run(cuda_device, 3, 4, 2, 64, 512, 3, kv_valid=[512, 130, 0]))


FLT_MAX = torch.finfo(torch.float32).max


def same_where_not_finite(got, ref, name):
    got, ref = got.double().cpu(), ref.double()
    for kind, at in (("nan", torch.isnan), ("+inf", torch.isposinf), ("-inf", torch.isneginf)):
        assert torch.equal(at(got), at(ref)), (name, kind)
    # column by column, since the columns of the largest values are 38 orders of magnitude above the others
    fin = torch.isfinite(ref)
    err = torch.where(fin, got - ref, 0.).flatten(0, -2).norm(dim=0) / torch.where(fin, ref, 0.).flatten(0, -2).norm(dim=0).clamp_min(1e-30)
    return err.max().item()


def extreme_inputs(dtype):
    q, k, v, do = orc.make_inputs(1, 4, 2, 70, 300, 128, 4, dtype)
    largest = torch.finfo(dtype).max
    q[..., 0] = q[..., 0].abs() + 0.1
    k[0, 1, 7, 0] = float("-inf")            # a key that scores -inf against every query
    v[0, 0, 3, 5] = float("inf")
    v[0, 0, 4, 6] = -largest
    v[0, 0, 9, 7] = largest
    v[0, 1, 70, 8] = float("-inf")
    v[0, 1, 71, 9] = float("nan")
    do[0, 1, 20, 10] = float("inf")
    do[0, 1, 21, 11] = largest
    do[0, 3, 66, 12] = float("-inf")
    do[0, 3, 67, 13] = float("nan")
    return q, k, v, do


def test_infinite_and_largest_values(cuda_device):
    """Infinities, NaN and the largest finite values come out where a plain sum has them, and spoil no other column: the
    split into tf32 parts must not round a finite value to infinity, nor turn an infinity into inf - inf."""
    import lv_xattn_b200 as lvx
    q, k, v, do = extreme_inputs(torch.float32)
    q6, k6, v6, do6 = (t.double() for t in (q, k, v, do))
    k6, v6 = k6.repeat_interleave(2, 1), v6.repeat_interleave(2, 1)
    p6 = (q6 @ k6.transpose(-1, -2) * SCALE).softmax(-1)
    # a zero probability times an infinity or NaN would be NaN: key 7 of head 1 has neither
    o6 = p6 @ v6
    qd, kd, vd, dod = (t.to(cuda_device) for t in (q, k, v, do))
    _, _, _, o, L = lvx._attn_forward(qd, kd, vd, False, SCALE, None)
    assert torch.isfinite(L).all()
    assert same_where_not_finite(o, o6, "o") <= 1e-5
    # dV = P^T dO sees dO only; the other gradients are NaN throughout as soon as one delta is infinite
    _, dk, dv = lvx._attn_backward(dod, qd, kd, vd, torch.zeros_like(qd), L, False, SCALE, None, "flash")
    dv6 = (p6.transpose(-1, -2) @ do6).view(1, 2, 2, 300, 128).sum(2)
    dv6[0, 1, 7] = 0                         # P = 0 there: 0 * inf is NaN in both, in the columns of head 3's extremes
    dv[0, 1, 7] = 0
    assert same_where_not_finite(dv, dv6, "dv") <= 1e-5


def test_largest_values_in_every_gradient(cuda_device):
    """A key and a query (of the second of three row tiles) with the largest value, each against zeros: finite everywhere, and
    dQ, which leaves tile by tile, must be complete and added once."""
    import lv_xattn_b200 as lvx
    q, k, v, do = orc.make_inputs(1, 4, 2, 70, 300, 128, 6, torch.float32)
    q[..., 14], k[..., 16] = 0, 0
    k[0, 0, 9, 14] = FLT_MAX
    q[0, 1, 40, 16] = FLT_MAX
    q6, k6, v6 = (t.double().requires_grad_() for t in (q, k, v))
    o6 = (q6 @ k6.repeat_interleave(2, 1).transpose(-1, -2) * SCALE).softmax(-1) @ v6.repeat_interleave(2, 1)
    grads6 = torch.autograd.grad(o6, (q6, k6, v6), do.double())
    qd, kd, vd, dod = (t.to(cuda_device) for t in (q, k, v, do))
    _, _, _, o, L = lvx._attn_forward(qd, kd, vd, False, SCALE, None)
    assert same_where_not_finite(o, o6.detach(), "o") <= 1e-5
    grads = lvx._attn_backward(dod, qd, kd, vd, o, L, False, SCALE, None, "flash")
    for name, got, ref in zip(("dq", "dk", "dv"), grads, grads6):
        assert same_where_not_finite(got, ref, name) <= 1e-5, name


def test_infinite_gradients_of_biased_fp16(cuda_device):
    """The same of the kernel's 16-bit form, whose inputs are tf32 as they stand: dV = P^T dO."""
    from lv_xattn_b200 import ops
    q, k, v, do = extreme_inputs(torch.float16)
    k, v = k.nan_to_num(posinf=0, neginf=0), v.nan_to_num(nan=0, posinf=0, neginf=0).clamp(-2, 2)
    bias = torch.randn(1, 1, 70, 300, generator=torch.Generator().manual_seed(5))
    p6 = (q.double() @ k.double().repeat_interleave(2, 1).transpose(-1, -2) * SCALE + bias.double()).softmax(-1)
    dv6 = (p6.transpose(-1, -2) @ do.double()).view(1, 2, 2, 300, 128).sum(2)
    qd, kd, vd, dod, bd = (t.to(cuda_device) for t in (q, k, v, do, bias))
    _, lse = ops.fwd_block(qd, kd, vd, SCALE, bias=bd)
    dq = torch.zeros(1, 4, 70, 128, device=cuda_device)
    dk, dv = torch.empty(1, 2, 300, 128, device=cuda_device), torch.empty(1, 2, 300, 128, device=cuda_device)
    ops.bwd_block(qd, dod, lse, torch.zeros(4, 70, device=cuda_device), kd, vd, SCALE, dq, dk, dv, False, bias=bd)
    assert same_where_not_finite(dv, dv6, "dv") <= 1e-5
