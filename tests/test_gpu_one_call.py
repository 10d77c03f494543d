"""The single-GPU passes that are one library call each: the same results as the step loop's own calls (which run while
kernel times are recorded), key-padding lengths in every form, and a wait that ran out noticed at the next call."""
import math

import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu
SCALE = 1.0 / math.sqrt(128.0)


def both_passes(q, k, v, do, **kw):
    import lv_xattn_b200 as lvx
    _, _, _, o, L = lvx._attn_forward(q, k, v, False, SCALE, None, **kw)
    return (o, L, *lvx._attn_backward(do, q, k, v, o, L, False, SCALE, None, "flash", **kw))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("case", ["plain", "padded", "bias", "no_keys"])
def test_same_as_the_separate_calls(cuda_device, case, dtype):
    from lv_xattn_b200 import ops
    B, Hq, Hkv, Sq, Skv = 2, 4, 2, 37, 0 if case == "no_keys" else 300
    q, k, v, do = (t.to(cuda_device) for t in orc.make_inputs(B, Hq, Hkv, Sq, max(Skv, 1), 128, 81, dtype))
    k, v = k[:, :, :Skv], v[:, :, :Skv]
    kw = {}
    if case == "padded":
        kw["kv_valid_len"] = [300, 129]
    if case == "bias":
        table = torch.randn(1, 1, Sq, Skv, device=cuda_device)
        kw.update(bias_func=lambda t: t, local_bias_args=[table], remote_bias_args=[])
    one = both_passes(q, k, v, do, **kw)
    ops.set_profiling(True)
    try:
        parts = both_passes(q, k, v, do, **kw)
    finally:
        ops.set_profiling(False)
    torch.cuda.synchronize()
    for name, a, b in zip(("o", "lse", "dq", "dk", "dv"), one, parts):
        assert a.dtype == b.dtype and a.shape == b.shape, name
        if name == "dq" and a.numel():
            # summed by reduce-adds in any order: 2^-20 of the largest value in fp32, one rounding of the result in 16 bits
            tol = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10, torch.float32: 2.0 ** -20}[dtype]
            assert (a.float() - b.float()).abs().max() <= tol * a.float().abs().max(), name
        else:
            assert torch.equal(a, b), name


def test_lengths_in_every_form(cuda_device):
    B, Skv = 300, 40                     # more entries than one launch of the length kernel takes
    q, k, v, do = (t.to(cuda_device) for t in orc.make_inputs(B, 1, 1, 2, Skv, 128, 82, torch.bfloat16))
    lens = [(7 * i) % 55 - 5 for i in range(B)]          # below 0 and above Skv among them
    ref = both_passes(q, k, v, do, kv_valid_len=torch.tensor(lens, device=cuda_device))
    for form in (lens, torch.tensor(lens, dtype=torch.int32), torch.tensor(lens, device=cuda_device, dtype=torch.int32)):
        got = both_passes(q, k, v, do, kv_valid_len=form)
        for i in (0, 1, 3, 4):
            assert torch.equal(got[i], ref[i])
    with pytest.raises(ValueError):
        both_passes(q, k, v, do, kv_valid_len=lens[:-1])


def test_a_wait_that_ran_out_is_noticed_at_the_next_call(cuda_device):
    """A flag that nothing sets, with the limit at 1 ms, leaves its code in the status word; the pass after it finds the
    word set and writes the host's copy."""
    import lv_xattn_b200 as lvx
    from lv_xattn_b200 import ops, _lib, peer_memory as pm
    from lv_xattn_b200.async_communication import P2PTimeoutError
    q, k, v, do = (t.to(cuda_device) for t in orc.make_inputs(1, 2, 1, 8, 128, 128, 83, torch.bfloat16))
    good = both_passes(q, k, v, do)
    flags = torch.zeros(8 * 16, dtype=torch.int32, device=cuda_device)
    lib = _lib.load()
    lib.lvx_p2p_set_timeout(0.001)
    try:
        ops.p2p_wait(flags, 1, 0, 1)
        lvx._attn_forward(q, k, v, False, SCALE, None)    # finds the word set, computes nothing and tells the host
        torch.cuda.synchronize()
        with pytest.raises(P2PTimeoutError):
            lvx._attn_forward(q, k, v, False, SCALE, None)
        again = both_passes(q, k, v, do)                  # raising has cleared the word
        assert torch.equal(good[0], again[0])
        ops.p2p_wait(flags, 1, 0, 1)
        lvx._attn_backward(do, q, k, v, good[0], good[1], False, SCALE, None, "flash")
        with pytest.raises(P2PTimeoutError):
            pm.check_device_status()
        pm.check_device_status()
    finally:
        lib.lvx_p2p_set_timeout(120.0)
        _lib.device_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("bias", [False, True])
def test_a_pass_that_found_the_word_set_is_reported(cuda_device, dtype, bias):
    """Either pass of every type, each as the first one after the wait: what it left unwritten must not go unnoticed."""
    import lv_xattn_b200 as lvx
    from lv_xattn_b200 import ops, _lib, peer_memory as pm
    from lv_xattn_b200.async_communication import P2PTimeoutError
    q, k, v, do = (t.to(cuda_device) for t in orc.make_inputs(1, 2, 1, 70, 300, 128, 84, dtype))
    kw = {}
    if bias:
        kw.update(bias_func=lambda t: t, local_bias_args=[torch.randn(1, 1, 70, 300, device=cuda_device)], remote_bias_args=[])
    good = both_passes(q, k, v, do, **kw)
    pm.check_device_status()
    flags = torch.zeros(8 * 16, dtype=torch.int32, device=cuda_device)
    lib = _lib.load()
    lib.lvx_p2p_set_timeout(0.001)
    try:
        for backward in (True, False):
            ops.p2p_wait(flags, 1, 0, 1)
            if backward:
                lvx._attn_backward(do, q, k, v, good[0], good[1], False, SCALE, None, "flash", **kw)
            else:
                lvx._attn_forward(q, k, v, False, SCALE, None, **kw)
            with pytest.raises(P2PTimeoutError):
                pm.check_device_status()
            pm.check_device_status()
        assert torch.equal(both_passes(q, k, v, do, **kw)[0], good[0])
    finally:
        lib.lvx_p2p_set_timeout(120.0)
        _lib.device_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_two_threads_on_two_streams(cuda_device, dtype):
    """Scratch is a call's own: passes that two threads launch at the same time, each on its own stream, give what they give
    one after the other (dQ up to the order of its additions)."""
    import threading
    shapes = [(1, 8, 2, 96, 3000), (2, 4, 2, 40, 1500)]
    inputs = [[t.to(cuda_device) for t in orc.make_inputs(*s, 128, 85 + i, dtype)] for i, s in enumerate(shapes)]
    alone = [both_passes(*x) for x in inputs]
    torch.cuda.synchronize()
    got = [[], []]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(30):
                got[i].append(both_passes(*inputs[i]))
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
    for i in range(2):
        assert len(got[i]) == 30
        for outs in got[i]:
            for name, a, b in zip(("o", "lse", "dq", "dk", "dv"), outs, alone[i]):
                if name == "dq":
                    assert (a.float() - b.float()).abs().max() <= tol * b.float().abs().max()
                else:
                    assert torch.equal(a, b), name


def test_captured_passes_keep_their_scratch(cuda_device):
    """Passes captured into a graph, then larger ones outside of it, then the graph again with new inputs."""
    q, k, v, do = (t.to(cuda_device) for t in orc.make_inputs(1, 8, 2, 50, 2000, 128, 87, torch.bfloat16))
    both_passes(q, k, v, do)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = both_passes(q, k, v, do)
    big = [t.to(cuda_device) for t in orc.make_inputs(1, 8, 2, 700, 9000, 128, 88, torch.bfloat16)]
    both_passes(*big)
    for seed in (89, 90):
        for old, new in zip((q, k, v, do), orc.make_inputs(1, 8, 2, 50, 2000, 128, seed, torch.bfloat16)):
            old.copy_(new)
        both_passes(*big)
        graph.replay()
        torch.cuda.synchronize()
        want = both_passes(q, k, v, do)
        for name, a, b in zip(("o", "lse", "dq", "dk", "dv"), outs, want):
            if name == "dq":
                assert (a.float() - b.float()).abs().max() <= 2.0 ** -8 * b.float().abs().max()
            else:
                assert torch.equal(a, b), name
