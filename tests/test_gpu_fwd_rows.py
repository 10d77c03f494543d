"""The forward kernel for few packed query rows (g * Sq <= 64) at the edges of its tiles: 16-row groups, 128-key tiles,
key ranges that are empty or end inside a tile, scores that force a rescale. Bars as in test_gpu_fwd.py."""
import math

import pytest
import torch

import _parity
from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu
SCALE = 1.0 / math.sqrt(128.0)


def run_and_check(device, B, Hq, Hkv, Sq, Skv, dtype, valid=None, gain=1.0, label=""):
    from lv_xattn_b200 import ops, _lib
    q, k, v, _ = orc.make_inputs(B, Hq, Hkv, Sq, Skv, 128, 11, dtype)
    q = q * gain
    o_ref, lse_ref = orc.attention_fwd(q, k, v, SCALE, valid)
    kvl = None if valid is None else torch.tensor(valid, dtype=torch.int32, device=device)
    o, lse = ops.fwd_block(q.to(device), k.to(device), v.to(device), SCALE, kv_valid_len=kvl)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    _parity.assert_lse_close(lse.cpu().view(B, Hq, Sq), lse_ref, label)
    _parity.assert_close(o.float().cpu(), o_ref, "o", label, *_parity.BF16["o"])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,Sq", [((1, 1), 1), ((4, 1), 4), ((1, 1), 17), ((4, 2), 16), ((3, 1), 11), ((4, 1), 16),
                                      ((5, 1), 13)])      # 1, 16, 17, 32, 33, 64 and 65 (the other kernel) rows
def test_row_groups(cuda_device, heads, Sq, dtype):
    run_and_check(cuda_device, 2, heads[0], heads[1], Sq, 1601, dtype, label=f"rows{heads}{Sq}{dtype}")


@pytest.mark.parametrize("skv", [1, 15, 127, 128, 129, 5 * 128 + 77, 40961])
def test_key_edges(cuda_device, skv):
    run_and_check(cuda_device, 1, 8, 2, 3, skv, torch.bfloat16, label=f"rows_keys{skv}")


@pytest.mark.parametrize("Sq", [2, 8, 16])
def test_key_padding_and_large_scores(cuda_device, Sq):
    # a sample without any valid key, ranges that end inside a warp's keys; queries scaled so that the running max jumps
    run_and_check(cuda_device, 4, 4, 1, Sq, 900, torch.bfloat16, valid=[900, 0, 387, 5], gain=16.0, label=f"rows_pad{Sq}")


@pytest.mark.parametrize("skv", [100, 5000])
def test_word_already_set(cuda_device, skv):
    """A wait that ran out earlier (a flag that nothing sets, with the limit at 1 ms) has left its code in the status word:
    the whole kernel leaves at once and writes nothing, and works again once the word has been cleared."""
    from lv_xattn_b200 import ops, _lib
    q, k, v, _ = (t.to(cuda_device) for t in orc.make_inputs(2, 8, 2, 5, skv, 128, 12, torch.bfloat16))
    o, lse = ops.fwd_block(q, k, v, SCALE)
    lib = _lib.load()
    lib.lvx_p2p_set_timeout(0.001)
    try:
        ops.p2p_wait(torch.zeros(8 * 16, dtype=torch.int32, device=cuda_device), 1, 0, 1)
        part = ops.fwd_partials(q, k, v, SCALE)
        part.ws.fill_(7)
        ops.fwd_partials(q, k, v, SCALE)
        torch.cuda.synchronize()
        assert (part.ws == 7).all()
    finally:
        lib.lvx_p2p_set_timeout(120.0)
        assert _lib.device_status() != 0                 # reading clears it
    again = ops.fwd_block(q, k, v, SCALE)
    assert torch.equal(again[0], o) and torch.equal(again[1], lse)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_infinities_and_nan(cuda_device, dtype):
    """Those of V come out in the columns where a plain sum has them, and a key that scores -inf counts as no key."""
    from lv_xattn_b200 import ops
    q, k, v, _ = orc.make_inputs(1, 6, 3, 7, 700, 128, 13, dtype)
    q[..., 0] = q[..., 0].abs() + 0.125
    k[0, 0, 130, 0] = float("-inf")
    v[0, 0, 3, 5] = float("inf")
    v[0, 1, 300, 6] = float("-inf")
    v[0, 1, 301, 7] = float("nan")
    k6, v6 = (t.double().repeat_interleave(2, 1) for t in (k, v))
    o6 = (q.double() @ k6.transpose(-1, -2) * SCALE).softmax(-1) @ v6
    o, lse = ops.fwd_block(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), SCALE)
    o = o.double().cpu()
    for at in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(at(o), at(o6))
    fin = torch.isfinite(o6)
    _parity.assert_close(o[fin], o6[fin], "o", f"rows_extremes{dtype}", *_parity.BF16["o"])
    assert torch.isfinite(lse).all()
