"""K/V projection of the visual states for the patched cross-attention layer.

The reference's `project()` closure (test_llama3.py:394-419) runs k_proj and v_proj on the visual states, reshapes
and transposes both to [B, H, S, D], expands them to the query head count and applies k_norm -- as separate torch
modules, in forward and again in the backward recompute. At the Llama-3.2-Vision shapes these GEMMs cost about as much
as the attention itself. `KVProjectFunc` is the same computation as ONE tensor-core GEMM with the per-head RMSNorm
fused into its epilogue and the result written directly in the [B, Hkv, S, 128] layout the attention kernels read
(`lvx_kv_project`). Its backward keeps the weight gradients on library GEMMs (torch.mm): one small kernel of this
library (`lvx_kv_project_grad_rows`) takes dK and dV from the attention's head-major layout to one row per key, with the
norm's backward on the way, and dWk = dK^T X and dWv = dV^T X are then one plain product each over all keys of the batch.
The states get a gradient only if they ask for one.
"""
from __future__ import annotations

import torch

from . import ops


class KVProjectFunc(torch.autograd.Function):
    """(states [B,S,hidden], wk, wv [Hkv*128, hidden], norm_weight [128], eps, n_kv_heads) -> (K, V) [B,Hkv,S,128]."""

    @staticmethod
    def forward(ctx, states, wk, wv, norm_weight, eps, n_kv_heads):
        k, v, rstd = ops.kv_project(states, wk, wv, norm_weight, eps, n_kv_heads)
        ctx.save_for_backward(states, wk, wv, norm_weight, k, rstd)
        ctx.n_kv_heads = n_kv_heads
        return k, v

    @staticmethod
    def backward(ctx, dk, dv):
        states, wk, wv, norm_weight, k, rstd = ctx.saved_tensors
        hid = states.shape[-1]
        want_x, want_wk, want_wv, want_nw = ctx.needs_input_grad[:4]
        dk_rows, dv_rows, dnw = ops.kv_grad_rows(k, dk, dv, rstd, norm_weight, want_x or want_wk, want_x or want_wv, want_nw)
        dk_rows, dv_rows = (None if t is None else t.flatten(0, 1) for t in (dk_rows, dv_rows))      # [B*S, Hkv*128]
        g_wk = g_wv = g_states = g_nw = None
        x = states.reshape(-1, hid)
        if want_wk:
            g_wk = torch.mm(dk_rows.t(), x)
        if want_wv:
            g_wv = torch.mm(dv_rows.t(), x)
        if want_x:
            g_states = (torch.mm(dk_rows, wk) + torch.mm(dv_rows, wv)).view(states.shape)
        if norm_weight is not None and want_nw:
            g_nw = dnw.to(norm_weight.dtype)
        return g_states, g_wk, g_wv, g_nw, None, None


def kv_project(states, wk, wv, norm_weight, eps, n_kv_heads):
    """The fused projection when the tensors qualify (CUDA, bf16/fp16, hidden a multiple of 64, an even number of KV
    heads); None otherwise, and the caller keeps its own modules."""
    if not ops.kv_project_supported(states, wk, wv, n_kv_heads):
        return None
    return KVProjectFunc.apply(states, wk, wv, norm_weight, float(eps), n_kv_heads)
