"""The tensor-core form of the biased blocks: every stride and shape that its loads distinguish, masks of -inf and of the
type's lowest value, rows without any key, and what its two-part P and dS keep of the fp32 values they stand for."""
import math

import pytest
import torch

import _parity
from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu
SCALE = 1.0 / math.sqrt(128.0)


def bias_of(kind, B, Hq, Sq, Skv, device):
    g = torch.Generator().manual_seed(5)
    if kind == "shared":                                   # one row per query, every head alike
        return torch.randn(1, 1, Sq, Skv, generator=g).to(device)
    if kind == "per_head":
        return torch.randn(B, Hq, Sq, Skv, generator=g).to(device)
    if kind == "keys":                                     # query stride 0
        return torch.randn(B, 1, 1, Skv, generator=g).to(device)
    if kind == "queries":                                  # key stride 0
        return torch.randn(B, 1, Sq, 1, generator=g).to(device)
    if kind == "transposed":                               # key stride > 1
        return torch.randn(1, 1, Skv, Sq, generator=g).to(device).transpose(2, 3)
    if kind == "offset":                                   # rows that start off a 16-byte boundary
        return torch.randn(1, 1, Sq, Skv + 1, generator=g).to(device)[..., 1:]
    b = torch.zeros(1, 1, Sq, Skv)
    b[..., Skv // 3:] = torch.finfo(torch.float32).min if kind == "lowest" else float("-inf")
    b[:, :, Sq // 2] = float("-inf")                       # a query that sees nothing
    return b.to(device)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["shared", "per_head", "keys", "queries", "transposed", "offset", "lowest", "masked"])
@pytest.mark.parametrize("shape", [(2, 4, 2, 77, 388), (1, 8, 1, 5, 129), (1, 2, 2, 300, 1024)])
def test_bias_forms(cuda_device, shape, kind, dtype):
    from lv_xattn_b200 import ops, _lib
    B, Hq, Hkv, Sq, Skv = shape
    q, k, v, do = orc.make_inputs(B, Hq, Hkv, Sq, Skv, 128, 71, dtype)
    bias = bias_of(kind, B, Hq, Sq, Skv, cuda_device)
    valid = [Skv - 3, Skv // 2][:B]
    bias_ref, do_ref = bias.cpu().expand(B, bias.shape[1], Sq, Skv), do.clone()
    if kind in ("lowest", "masked"):
        # the oracle gets the query that sees nothing as one without a gradient; its output is zero and its lse -inf
        bias_ref = bias_ref.clone()
        bias_ref[:, :, Sq // 2] = 0
        do_ref[:, :, Sq // 2] = 0
    ref = orc.attention_fwd_bwd(q, k, v, do_ref, SCALE, valid, bias=bias_ref)
    if kind in ("lowest", "masked"):
        ref[0][:, :, Sq // 2] = 0
        ref[1][:, :, Sq // 2] = float("-inf")
    qd, kd, vd, dod = (t.to(cuda_device) for t in (q, k, v, do))
    kvl = torch.tensor(valid, dtype=torch.int32, device=cuda_device)
    o, lse = ops.fwd_block(qd, kd, vd, SCALE, kv_valid_len=kvl, bias=bias)
    delta = ops.bwd_prep(o, dod)
    dq = torch.zeros(B, Hq, Sq, 128, device=cuda_device)
    dk, dv = torch.empty_like(kd), torch.empty_like(vd)
    ops.bwd_block(qd, dod, lse, delta, kd, vd, SCALE, dq, dk, dv, "final", kvl, bias=bias)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    label = f"bias_{kind}{shape}{dtype}"
    _parity.assert_lse_close(lse.cpu().view(B, Hq, Sq), ref[1], label)
    _parity.assert_close(o.float().cpu(), ref[0], "o", label, *_parity.BF16["o"])
    _parity.assert_grads_16bit((dq, dk, dv), ref[2:], label)


@pytest.mark.parametrize("shape", [(2, 4, 2, 77, 388), (1, 2, 2, 300, 200), (1, 1, 1, 64, 130), (1, 3, 1, 96, 129)])
def test_last_tile_reads_no_bias_of_rows_that_do_not_exist(cuda_device, shape):
    """The packed rows end inside a 128-row tile. The per-head bias is a leading slice of a larger buffer of NaN, so that a
    value read past the last head's rows shows in dK and dV (a NaN P times a zero dO)."""
    from lv_xattn_b200 import ops, _lib
    B, Hq, Hkv, Sq, Skv = shape
    q, k, v, do = orc.make_inputs(B, Hq, Hkv, Sq, Skv, 128, 75, torch.bfloat16)
    n = B * Hq * Sq * Skv
    buf = torch.full((n + 256 * Skv,), float("nan"))
    bias = buf[:n].view(B, Hq, Sq, Skv)
    bias.copy_(torch.randn(B, Hq, Sq, Skv, generator=torch.Generator().manual_seed(76)))
    ref = orc.attention_fwd_bwd(q, k, v, do, SCALE, None, bias=bias)
    bias = buf.to(cuda_device)[:n].view(B, Hq, Sq, Skv)
    qd, kd, vd, dod = (t.to(cuda_device) for t in (q, k, v, do))
    o, lse = ops.fwd_block(qd, kd, vd, SCALE, bias=bias)
    delta = ops.bwd_prep(o, dod)
    dq = torch.zeros(B, Hq, Sq, 128, device=cuda_device)
    dk, dv = torch.empty_like(kd), torch.empty_like(vd)
    ops.bwd_block(qd, dod, lse, delta, kd, vd, SCALE, dq, dk, dv, "final", None, bias=bias)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    _parity.assert_close(o.float().cpu(), ref[0], "o", f"bias_tail{shape}", *_parity.BF16["o"])
    _parity.assert_grads_16bit((dq, dk, dv), ref[2:], f"bias_tail{shape}")


def test_two_part_operands(cuda_device):
    """fp32 outputs against 64 bits. P and dS are held to 2^-17 of each value (two bf16 numbers), the scores to fp32 sums
    over 128 products; 2^-15 leaves a factor of four. One bf16 rounding would show at 2^-9."""
    from lv_xattn_b200 import ops
    B, Hq, Hkv, Sq, Skv = 1, 4, 2, 160, 1000
    q, k, v, do = orc.make_inputs(B, Hq, Hkv, Sq, Skv, 128, 73, torch.bfloat16)
    bias = torch.randn(1, 1, Sq, Skv, generator=torch.Generator().manual_seed(74))
    q6, k6, v6, do6 = (t.double().requires_grad_() for t in (q, k, v, do))
    s = q6 @ k6.repeat_interleave(2, 1).transpose(-1, -2) * SCALE + bias.double()
    o6 = s.softmax(-1) @ v6.repeat_interleave(2, 1)
    dq6, dk6, dv6 = torch.autograd.grad(o6, (q6, k6, v6), do6)
    d = cuda_device
    qd, kd, vd, dod, bd = (t.to(d) for t in (q, k, v, do, bias))
    o, lse = ops.fwd_block(qd, kd, vd, SCALE, final=False, bias=bd)
    delta = (o6.detach() * do6.detach()).sum(-1).float().view(Hq, Sq).to(d)
    dq = torch.zeros(B, Hq, Sq, 128, device=d)
    dk, dv = torch.empty(B, Hkv, Skv, 128, device=d), torch.empty(B, Hkv, Skv, 128, device=d)
    ops.bwd_block(qd, dod, lse, delta, kd, vd, SCALE, dq, dk, dv, False, bias=bd)
    for name, got, ref in (("o", o, o6), ("dq", dq, dq6), ("dk", dk, dk6), ("dv", dv, dv6)):
        err = ((got.cpu().double() - ref).norm() / ref.norm()).item()
        assert err <= 2.0 ** -15, (name, err)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("below", [18.3, 25.5])
@pytest.mark.parametrize("at", [0, 700, 5999])
def test_small_probabilities_beside_a_dominant_key(cuda_device, dtype, below, at):
    """One key, whose value is zero, outweighs every other one by 2^18 or 2^25: the output is what the others add up to.
    In fp16, P relative to the row's maximum would be subnormal or nothing there. P is held to 2^-25 of 2^-12 of the
    maximum, i.e. to 2^-11.5 of the smaller probabilities here, and the output is rounded to 16 bits."""
    from lv_xattn_b200 import ops
    B, H, Sq, Skv = 1, 2, 40, 6000
    g = torch.Generator().manual_seed(77)
    q = torch.zeros(B, H, Sq, 128, dtype=dtype)
    k = torch.empty(B, H, Skv, 128).normal_(0, 0.5, generator=g).to(dtype)
    v = (1 + torch.empty(B, H, Skv, 128).normal_(0, 0.5, generator=g)).to(dtype)
    v[:, :, at] = 0
    bias = torch.full((1, 1, Sq, Skv), -below * math.log(2.0))
    bias[..., at] = 0
    ref = bias.double().expand(B, H, Sq, Skv).softmax(-1) @ v.double()
    o, lse = ops.fwd_block(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), SCALE, bias=bias.to(cuda_device))
    err = ((o.cpu().double() - ref).norm() / ref.norm()).item()
    assert err <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10), err
    assert (lse.cpu().double() - torch.logsumexp(bias.double()[0, 0], -1)).abs().max() <= 1e-5


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_infinite_values_and_gradients(cuda_device, dtype):
    """An infinite V gives its column of O, and an infinite dO its column of dV, the infinity that a plain sum gives them, and
    NaN stays in its column: the second part of P, which may be zero or negative, must not turn them into NaN. A -inf key
    is no key."""
    from lv_xattn_b200 import ops
    B, Hq, Hkv, Sq, Skv = 1, 4, 2, 150, 700
    q, k, v, do = orc.make_inputs(B, Hq, Hkv, Sq, Skv, 128, 78, dtype)
    q[..., 0] = q[..., 0].abs() + 0.125
    k[0, 1, 400, 0] = float("-inf")
    v[0, 0, 3, 5] = float("inf")
    v[0, 0, 690, 6] = float("-inf")
    v[0, 1, 301, 7] = float("nan")
    do[0, 1, 20, 8] = float("inf")
    do[0, 2, 149, 9] = float("-inf")
    do[0, 3, 40, 10] = float("nan")
    bias = torch.randn(1, 1, Sq, Skv, generator=torch.Generator().manual_seed(79))
    k6, v6 = (t.double().repeat_interleave(2, 1) for t in (k, v))
    p6 = (q.double() @ k6.transpose(-1, -2) * SCALE + bias.double()).softmax(-1)
    o6 = p6 @ v6
    dv6 = (p6.transpose(-1, -2) @ do.double()).view(1, 2, 2, Skv, 128).sum(2)
    qd, kd, vd, dod, bd = (t.to(cuda_device) for t in (q, k, v, do, bias))
    o, lse = ops.fwd_block(qd, kd, vd, SCALE, bias=bd)
    dq = torch.zeros(B, Hq, Sq, 128, device=cuda_device)
    dk, dv = torch.empty_like(kd), torch.empty_like(vd)
    ops.bwd_block(qd, dod, lse, torch.zeros(B * Hq, Sq, device=cuda_device), kd, vd, SCALE, dq, dk, dv, "final", bias=bd)
    dv[0, 1, 400] = dv6[0, 1, 400] = 0       # no key: 0 * inf there
    for name, got, ref in (("o", o, o6), ("dv", dv, dv6)):
        got = got.double().cpu()
        for at in (torch.isnan, torch.isposinf, torch.isneginf):
            assert torch.equal(at(got), at(ref)), (name, at.__name__)
        fin = torch.isfinite(ref)
        assert ((got - ref)[fin].norm() / ref[fin].norm()).item() <= 1e-2, name


@pytest.mark.parametrize("skv", [1, 31, 33, 64, 127, 128, 129, 252, 256, 257, 260, 383, 516])
@pytest.mark.parametrize("valid", [None, 0.6])
def test_staged_pieces_of_the_forward(cuda_device, skv, valid):
    """Aligned and unaligned rows on both sides of 256 keys, with ends inside a piece of 32 keys. The bias is followed by NaN,
    and its keys past the last valid one are NaN: neither may be seen."""
    from lv_xattn_b200 import ops
    B, H, Sq = 1, 2, 140
    q, k, v, _ = orc.make_inputs(B, H, H, Sq, skv, 128, 80, torch.bfloat16)
    n = None if valid is None else max(1, int(skv * valid))
    buf = torch.full((H * Sq * skv + 4096,), float("nan"))
    bias = buf[:H * Sq * skv].view(1, H, Sq, skv)
    bias.copy_(torch.randn(1, H, Sq, skv, generator=torch.Generator().manual_seed(81)))
    o_ref, lse_ref = orc.attention_fwd(q, k, v, SCALE, None if n is None else [n], bias=bias)
    if n is not None:
        bias[..., n:] = float("nan")
    kvl = None if n is None else torch.tensor([n], dtype=torch.int32, device=cuda_device)
    bias = buf.to(cuda_device)[:H * Sq * skv].view(1, H, Sq, skv)
    o, lse = ops.fwd_block(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), SCALE, kv_valid_len=kvl, bias=bias)
    _parity.assert_lse_close(lse.cpu().view(B, H, Sq), lse_ref, f"bias_pieces{skv}")
    _parity.assert_close(o.float().cpu(), o_ref, "o", f"bias_pieces{skv}", *_parity.BF16["o"])
