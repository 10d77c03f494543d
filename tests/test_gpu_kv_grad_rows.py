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
