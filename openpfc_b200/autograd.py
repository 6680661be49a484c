"""torch.autograd.Function over the hand-written adjoint (gradient harness only).

    psi_T = PfcEvolve.apply(psi0, r, model, n_steps, K)

runs the model's step `n_steps` times on the GPU with snapshots every K steps
(opfc_forward_checkpointed) and, on backward, the adjoint through the C ABI
(opfc_adjoint).  The model is any of the package's models with an adjoint
(plain, filtered, Tungsten, Aluminum without a moving gradient); psi0 and psi_T
are CUDA tensors in the model's precision with shape (N2, N1, N0); r is a 0-d
tensor for the models with r (plain, filtered) and None otherwise.  No torch
kernel is involved in either direction: torch only carries the buffers and the
autograd graph.
"""
from __future__ import annotations

import torch

from . import FP64, PfcB200


def _streams(model, t: torch.Tensor):
    """(the model's stream, torch's current one) for a device tensor, else None."""
    if not t.is_cuda:
        return None
    own = getattr(model, "_torch_stream", None)
    if own is None:
        own = model._torch_stream = torch.cuda.ExternalStream(model.stream, device=t.device)
    return own, torch.cuda.current_stream(t.device)


class PfcEvolve(torch.autograd.Function):
    @staticmethod
    def forward(ctx, psi0: torch.Tensor, r, model, n_steps: int, K: int = 20):
        if r is not None:
            model.set_r(float(r))
        psi0 = psi0.detach().contiguous()
        out = torch.empty_like(psi0)
        # the model works on a stream of its own: after what torch has queued for psi0
        # and on out's memory, and before what torch does with out
        s = _streams(model, psi0)
        if s:
            s[0].wait_stream(s[1])
        model.set_psi(psi0)
        model.forward_checkpointed(n_steps, K)
        model.get_psi(out)
        if s:
            s[1].wait_stream(s[0])
        ctx.model = model
        ctx.has_r = r is not None
        ctx.r_dtype = r.dtype if r is not None else None
        ctx.r_device = r.device if r is not None else None
        return out

    @staticmethod
    def backward(ctx, grad_out: torch.Tensor):
        grad_out = grad_out.detach().contiguous()
        g0 = torch.empty_like(grad_out)
        s = _streams(ctx.model, grad_out)
        if s:
            s[0].wait_stream(s[1])
        g0, gr, _ = ctx.model.adjoint(grad_out, g0)
        g_r = torch.tensor(gr, dtype=ctx.r_dtype, device=ctx.r_device) if ctx.has_r else None
        return g0, g_r, None, None, None


def make_model(n, dx, precision=FP64, dt=0.5, r=-0.25, device=0) -> PfcB200:
    m = PfcB200(n, dx, r=r, precision=precision, device=device)
    m.initialize(dt)
    return m
