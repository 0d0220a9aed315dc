"""The expert part of a mixture-of-experts layer as one autograd function: token rows into the expert-grouped matrix,
gate|up and down projections as grouped GEMMs with SwiGLU between them, weighted expert rows back to their tokens.

The row movement runs on ``cuda/moe_ops.cu``.  Between the kernels only the rows of used tiles carry values: padding
rows inside an expert's segment are zeroed (the weight-gradient GEMM runs over them), rows of unused tiles are never
read, so no buffer is cleared as a whole.
Reference: src/model/qwen3_5_text.cc:882-993.
"""
from __future__ import annotations

import torch

from .. import _native as nv
from .gemm import count_launch, gemm_raw, use_native
from .grouped_gemm import TILE_M


def supported(x: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor, top_k: int) -> bool:
    """bf16 CUDA rows whose widths allow 16-byte pieces and TMA, up to 256 experts and 32 experts per token."""
    E, two_i, H = gate_up.shape
    return (use_native(x) and gate_up.dtype == down.dtype == torch.bfloat16 and x.dim() == 2 and x.shape[0] > 0
            and H % 8 == 0 and (two_i // 2) % 8 == 0 and E <= 256 and 0 < top_k <= 32
            and gate_up.is_contiguous() and down.is_contiguous())


def _grouped(x, w, out, tile_group, *, b_mn):
    """``out = x @ w[expert].T`` (or ``x @ w[expert]`` with ``b_mn``) on the used 128-row tiles of ``x``."""
    E, rows, cols = w.shape
    M, K = x.shape
    N = out.shape[1]
    gemm_raw(x, w.view(E * rows, cols), out, M, N, K, a_mn=False, b_mn=b_mn, epi=nv.EPI_STORE_BF16,
             block_n=256 if N >= 256 else 128, tile_group=tile_group, b_group_rows=rows, b_total_rows=E * rows)


def _grouped_wgrad(dy, x, w, offsets):
    """``dw[e] += dy_e.T @ x_e`` into ``w.main_grad``, or a new tensor when the parameter has none."""
    E, N, K = w.shape
    main_grad = getattr(w, "main_grad", None)
    acc = main_grad if main_grad is not None else torch.zeros(w.shape, dtype=torch.float32, device=w.device)
    gemm_raw(dy, x, acc.view(E * N, K), N, K, dy.shape[0], a_mn=True, b_mn=True, epi=nv.EPI_ATOMIC_F32,
             block_n=256 if K >= 256 else 128, k_group_offsets=offsets, num_groups=E, c_group_stride=N * K)
    return None if main_grad is not None else acc.to(w.dtype)


class _MoeExperts(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, gate_up, down, layout):
        row, tile_group, offsets, m_pad, totals = layout
        T, H = x.shape
        k = w.shape[1]
        E, two_i, _ = gate_up.shape
        dev, lib, st = x.device, nv.cuda(), nv.stream()
        x = x.contiguous()
        if x.data_ptr() % 16:
            x = x.clone()
        w32 = w.float().contiguous()

        def rows(n):
            return torch.empty((m_pad, n), dtype=x.dtype, device=dev)
        xp, gu, act, yp = rows(H), rows(two_i), rows(two_i // 2), rows(H)
        nv.check(lib.cvb_moe_dispatch(x.data_ptr(), row.data_ptr(), xp.data_ptr(), offsets.data_ptr(),
                                      totals.data_ptr(), T, k, H, E, st), "cvb_moe_dispatch")
        _grouped(xp, gate_up, gu, tile_group, b_mn=False)
        nv.check(lib.cvb_swiglu_fwd(gu.data_ptr(), act.data_ptr(), m_pad, two_i // 2, two_i, st), "cvb_swiglu_fwd")
        _grouped(act, down, yp, tile_group, b_mn=False)
        out = torch.empty((T, H), dtype=x.dtype, device=dev)
        nv.check(lib.cvb_moe_combine(yp.data_ptr(), row.data_ptr(), w32.data_ptr(), out.data_ptr(), T, k, H, st),
                 "cvb_moe_combine")
        count_launch(4)
        ctx.save_for_backward(xp, gu, act, yp, w32, gate_up, down, row, tile_group, offsets, totals)
        ctx.w_dtype = w.dtype
        return out

    @staticmethod
    def backward(ctx, dout):
        xp, gu, act, yp, w32, gate_up, down, row, tile_group, offsets, totals = ctx.saved_tensors
        T, k = w32.shape
        m_pad, H = xp.shape
        E, two_i, _ = gate_up.shape
        dev, lib, st = dout.device, nv.cuda(), nv.stream()
        dout = dout.contiguous()
        if dout.data_ptr() % 16:
            dout = dout.clone()
        dyp = torch.empty_like(yp)
        dw = torch.empty_like(w32)
        nv.check(lib.cvb_moe_combine_bwd(dout.data_ptr(), yp.data_ptr(), row.data_ptr(), w32.data_ptr(),
                                         dyp.data_ptr(), dw.data_ptr(), offsets.data_ptr(), totals.data_ptr(), T, k, H,
                                         E, st), "cvb_moe_combine_bwd")
        dact = torch.empty_like(act)
        _grouped(dyp, down, dact, tile_group, b_mn=True)
        d_down = _grouped_wgrad(dyp, act, down, offsets) if ctx.needs_input_grad[3] else None
        dgu = torch.empty_like(gu)
        nv.check(lib.cvb_swiglu_bwd(dact.data_ptr(), gu.data_ptr(), dgu.data_ptr(), m_pad, two_i // 2, two_i, st),
                 "cvb_swiglu_bwd")
        d_gu = _grouped_wgrad(dgu, xp, gate_up, offsets) if ctx.needs_input_grad[2] else None
        dx = None
        count_launch(3)
        if ctx.needs_input_grad[0]:
            dxp = dyp                                   # same shape, no longer needed
            _grouped(dgu, gate_up, dxp, tile_group, b_mn=True)
            dx = torch.empty((T, H), dtype=xp.dtype, device=dev)
            nv.check(lib.cvb_moe_combine(dxp.data_ptr(), row.data_ptr(), None, dx.data_ptr(), T, k, H, st),
                     "cvb_moe_combine")
            count_launch()
        return dx, dw.to(ctx.w_dtype), d_gu, d_down, None


def moe_experts(x: torch.Tensor, expert_ids: torch.Tensor, weights: torch.Tensor, gate_up: torch.Tensor,
                down: torch.Tensor) -> torch.Tensor:
    """``out[t] = sum_j weights[t, j] * down[e] @ swiglu(gate_up[e] @ x[t])`` with ``e = expert_ids[t, j]``.

    x bf16 [T, H], expert_ids int64 [T, k], weights fp32 [T, k], gate_up [E, 2I, H], down [E, H, I] (see ``supported``).
    """
    from ..models.moe import expert_layout_native
    layout = expert_layout_native(expert_ids.reshape(-1).contiguous(), gate_up.shape[0], TILE_M)
    return _MoeExperts.apply(x, weights, gate_up, down, layout)
