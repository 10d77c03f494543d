"""lvx_kv_project_grad_rows: the norm's backward and the change of layout against lvx_knorm_bwd and a transpose, at sizes
around the 64 rows that a block takes at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("shape", [(1, 2, 1), (2, 4, 63), (1, 2, 64), (3, 2, 1601), (1, 8, 8192)])
def test_rows_layout(cuda_device, shape, norm, dtype):
    from lv_xattn_b200 import ops
    B, H, S = shape
    g = torch.Generator(device=cuda_device).manual_seed(3)
    k, dk, dv = (torch.empty(B, H, S, 128, device=cuda_device).normal_(0, 1, generator=g).to(dtype) for _ in range(3))
    rstd = torch.rand(B, H, S, device=cuda_device, generator=g) + 0.5
    w = (1 + 0.1 * torch.empty(128, device=cuda_device).normal_(0, 1, generator=g)).to(dtype) if norm else None
    dk_rows, dv_rows, dw = ops.kv_grad_rows(k, dk, dv, rstd, w)
    want, dw_ref = ops.knorm_bwd(k, dk, rstd, w) if norm else (dk, None)
    assert torch.equal(dk_rows.view(B, S, H, 128), want.transpose(1, 2))
    assert torch.equal(dv_rows.view(B, S, H, 128), dv.transpose(1, 2))
    if norm:
        # fp32 sums over B*H*S values of size about 1 in another order of additions
        assert (dw - dw_ref).abs().max() <= 2.0 ** -20 * B * H * S
    else:
        assert dw is None


@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("wants", [(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)])
def test_only_what_is_wanted(cuda_device, wants, norm):
    from lv_xattn_b200 import ops
    B, H, S = 2, 2, 131
    g = torch.Generator(device=cuda_device).manual_seed(4)
    k, dk, dv = (torch.empty(B, H, S, 128, device=cuda_device).normal_(0, 1, generator=g).bfloat16() for _ in range(3))
    rstd = torch.rand(B, H, S, device=cuda_device, generator=g) + 0.5
    w = torch.ones(128, device=cuda_device, dtype=torch.bfloat16) if norm else None
    whole = ops.kv_grad_rows(k, dk, dv, rstd, w)
    some = ops.kv_grad_rows(k, dk, dv, rstd, w, *(bool(x) for x in wants))
    for i, (a, b) in enumerate(zip(some, whole)):
        assert (a is None) == (not wants[i] or b is None)
        if a is not None and i < 2:
            assert torch.equal(a, b)
        elif a is not None:
            assert (a - b).abs().max() <= 2.0 ** -20 * B * H * S          # atomic additions in any order


@pytest.mark.parametrize("frozen", ["k", "v", "kv", "norm"])
def test_frozen_projections_cost_no_layout(cuda_device, frozen, monkeypatch):
    """The backward of the projection asks for the rows that a gradient will be made of, and the gradients are those of the
    whole backward."""
    from lv_xattn_b200 import ops
    from lv_xattn_b200.projection import KVProjectFunc
    g = torch.Generator(device=cuda_device).manual_seed(5)
    mk = lambda *sh, std=1.0: torch.empty(*sh, device=cuda_device).normal_(0, std, generator=g).bfloat16()
    tensors = dict(states=mk(2, 70, 128), wk=mk(256, 128, std=0.1), wv=mk(256, 128, std=0.1), nw=1 + 0.1 * mk(128))
    dk, dv = mk(2, 2, 70, 128), mk(2, 2, 70, 128)
    asked = []
    rows = ops.kv_grad_rows
    monkeypatch.setattr(ops, "kv_grad_rows", lambda *a: asked.append(rows(*a)) or asked[-1])

    def grads(names):
        t = {n: x.clone().requires_grad_(n in names) for n, x in tensors.items()}
        k, v = KVProjectFunc.apply(t["states"], t["wk"], t["wv"], t["nw"], 1e-5, 2)
        return dict(zip(names, torch.autograd.grad((k, v), [t[n] for n in names], (dk, dv))))

    names = [n for n, off in (("wk", "k" in frozen), ("wv", "v" in frozen), ("nw", frozen == "norm")) if not off]
    got = grads(names)
    assert [t is not None for t in asked[-1]] == ["wk" in names, "wv" in names, "nw" in names]
    want = grads(["wk", "wv", "nw"])
    for n in names:
        if n == "nw":
            assert (got[n] - want[n]).abs().max() <= 2.0 ** -8 * want[n].abs().max()
        else:
            assert torch.equal(got[n], want[n]), n
