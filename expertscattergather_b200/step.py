"""One explicit training step of the path: gather -> scatter -> loss = sum(Out * G) -> backward.

The six operator launches are issued directly (no autograd graph), in the order autograd would run them for
the reference's modules.  ``on_weight_grad(name, tensor)`` is called as soon as each weight gradient has been
enqueued, which is where a data-parallel caller starts that gradient's all-reduce so it overlaps the rest of
the backward pass.
"""
from __future__ import annotations

from typing import Callable, Optional

import torch

from . import ops

__all__ = ["train_step", "takes_fused_pairs"]



def _is_capturing(stream: "torch.cuda.Stream") -> bool:
    with torch.cuda.stream(stream):
        return bool(torch.cuda.is_current_stream_capturing())


def _prefilled_outputs(X: torch.Tensor, T: int, n_out: int, main: "torch.cuda.Stream"):
    """Allocates Out [B,T,n_out] and dX (like X) and zero-fills them on the fill stream; returns the two tensors, an
    event for "Out is filled" and one for "both are filled".

    The tensors come from the fill stream's own memory pool: nothing ties the fills to work already queued on the
    main stream (the tail of the previous step), so they run under it.  The scatters then add into the zeros.  Inside a
    stream capture the fill stream first joins the capture through the main stream."""
    dev = X.device
    fills = ops.fill_stream(dev)
    if _is_capturing(main) and not _is_capturing(fills):
        fills.wait_stream(main)
    with torch.cuda.stream(fills):
        Out = torch.empty((X.shape[0], T, n_out), device=dev, dtype=X.dtype)
        dX = torch.empty_like(X, memory_format=torch.contiguous_format)
        Out.record_stream(main)
        dX.record_stream(main)
        ops.fill_zero(Out)
        out_filled = fills.record_event()
        ops.fill_zero(dX)
    return Out, dX, out_filled, fills.record_event()


def takes_fused_pairs(X: torch.Tensor, Wg: torch.Tensor, Ind: torch.Tensor) -> bool:
    """Whether :func:`train_step` runs G -> S and dY -> dX as one fused kernel each for these tensors."""
    return ops.fused_pair_preferred(X, Wg, Ind)


def train_step(X: torch.Tensor, Wg: torch.Tensor, Ws: torch.Tensor, Ind: torch.Tensor, G: torch.Tensor,
               on_weight_grad: Optional[Callable[[str, torch.Tensor], None]] = None, overlap: bool = True,
               fused_pairs: bool = True) -> dict:
    """X [B,T,I], Wg [E,I,J], Ws [E,J,I], Ind [B,E,K], G [B,T,I] (the gradient of the loss w.r.t. Out).

    Returns Y, Out, dY, dX, dWg, dWs.  Equivalent to
    ``Y = ExpertGather(X, Ind); Out = ExpertScatter(Y, Ind, T); (Out*G).sum().backward()``.

    With ``overlap`` the two weight-gradient kernels, which are off the critical chain G -> S -> dY -> dX, run on a helper
    stream, each started as soon as its inputs exist.  With ``on_weight_grad`` (the data-parallel case) the operators
    stay on one stream in an order that puts both weight gradients, and with them the start of their reductions,
    before the last scatter; the zero fills of float32 outputs run beside them.  With ``fused_pairs`` float32 shapes that
    the fused pair kernel takes run G -> S and dY -> dX as one kernel each.
    """
    T = X.shape[1]
    if on_weight_grad is not None:
        # data-parallel order: both weight gradients come before the long dX scatter, so that the reductions the
        # callback starts (dW_s first, then dW_g) run behind the kernels that are still to come
        main = torch.cuda.current_stream(X.device)
        Out = dX = None
        if X.dtype == torch.float32:
            Out, dX, out_filled, fills_done = _prefilled_outputs(X, T, Ws.shape[2], main)
        Y = ops.gather_gemm(X, Wg, Ind, w_layout="cn")
        if Out is not None:
            main.wait_event(out_filled)
        Out = ops.gemm_scatter(Y, Ws, Ind, T, w_layout="cn", out=Out)
        dY = ops.gather_gemm(G, Ws, Ind, w_layout="nc")
        dWs = ops.dweight(G, Y, Ind, out_layout="direct_rows")
        on_weight_grad("Ws", dWs)
        dWg = ops.dweight(X, dY, Ind, out_layout="gathered_rows")
        on_weight_grad("Wg", dWg)
        if dX is not None:
            main.wait_event(fills_done)
        dX = ops.gemm_scatter(dY, Wg, Ind, T, w_layout="nc", out=dX)
        return {"Y": Y, "Out": Out, "dY": dY, "dX": dX, "dWg": dWg, "dWs": dWs}
    Y, Out, dY, dX, dWg, dWs = ops._host().train_step(X, Wg, Ws, Ind, G, overlap, fused_pairs)
    return {"Y": Y, "Out": Out, "dY": dY, "dX": dX, "dWg": dWg, "dWs": dWs}
