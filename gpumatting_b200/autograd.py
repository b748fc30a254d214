"""torch.autograd wrapper of the Levin matting solve and its adjoint.

alpha = levin_matte(image, gamma, s) assembles the Levin Laplacian of the
[0, 1] RGB image (Matting.cu:79-218 math, eps as a parameter), solves
(L + diag(gamma)) alpha = gamma * s on the GPU (multigrid-preconditioned CG
by default), and on backward runs gm_levin_adjoint: one more solve of the symmetric
system for lambda, then the window-statistics back-propagation to the image
and lambda * (s - alpha) for gamma.  The reference has no gradients; this is
the differentiable form of its cgSolve path (main.cu:458-526).
"""
from __future__ import annotations

import torch

from . import _lib as L
from . import api

# Stores of up to this size (0.7 Mpixel in FP16) are tensors of torch's caching
# allocator: a training loop makes one per step, and the driver's cudaMalloc and
# cudaFree of one take 0.4-0.6 ms (spikes of 10-20 ms were seen) of a step's 6 at
# 512x512.  That memory is ordered by the stream it was made on, which is right
# here and not for api.LevinStore: the solves and the adjoint of one node run on
# the stream that is current in its forward pass.  Next to the solves of a
# larger image the allocation is small (under 2 % at 1080p), and its memory goes
# back to the driver.
CACHED_STORE_BYTES = 64 << 20


class _CachedStore(api.LevinStore):
    """api.LevinStore over memory of torch's caching allocator."""

    def __init__(self, W: int, H: int, precision: str, memory):
        P, esize = (W + 7) // 8 * 8, 4 if precision == "fp32" else 2
        high, low, one = _plane_bytes(W, H, precision)
        self.memory = memory
        w32 = memory.data_ptr()
        w = w32 if esize == 4 else w32 + high
        gamma = w32 + high + low
        self.s = L.GmLevinStore(W, H, P, api.PRECISIONS[precision], w, w32, gamma, gamma + one, gamma + 2 * one,
                                gamma + 3 * one, 0, 0)
        self.W, self.H, self.precision = W, H, precision


def _plane_bytes(W: int, H: int, precision: str):
    """Bytes of the 12 FP32 planes, of the 12 two-byte ones and of one vector, in
    multiples of 256 as gm_levin_store_alloc lays them out."""
    n = (W + 7) // 8 * 8 * H
    return [(x + 255) // 256 * 256 for x in (48 * n, 0 if precision == "fp32" else 24 * n, 4 * n)]


def _new_store(W: int, H: int, precision: str) -> api.LevinStore:
    if W > 0 and H > 0 and precision in api.PRECISIONS:
        high, low, one = _plane_bytes(W, H, precision)
        size = high + low + 4 * one
        if size <= CACHED_STORE_BYTES:
            return _CachedStore(W, H, precision, torch.empty(size, dtype=torch.uint8, device="cuda"))
    return api.LevinStore(W, H, precision)


class LevinMatte(torch.autograd.Function):
    @staticmethod
    def forward(ctx, image, gamma, s, eps: float, precision: str, rtol: float, max_iters: int,
                adjoint_rtol: float, solver: str):
        if image.dim() != 3 or image.shape[2] != 3 or image.dtype != torch.float32 or not image.is_cuda:
            raise ValueError("image must be a CUDA float32 tensor of shape (H, W, 3)")
        H, W, _ = image.shape
        if gamma.shape != (H, W) or s.shape != (H, W):
            raise ValueError("gamma and s must be (H, W)")
        im4 = torch.zeros((H, W, 4), dtype=torch.float32, device=image.device)
        im4[..., :3] = image.detach()
        g = gamma.detach().to(torch.float32).contiguous()
        sv = s.detach().to(torch.float32).contiguous()
        store = _new_store(W, H, precision).assemble(im4, gamma_map=g, s_map=sv, eps=eps)
        alpha = torch.full((H, W), 0.5, dtype=torch.float32, device=image.device)
        res = store.solve(alpha, solver, rtol=rtol, max_iters=max_iters)
        ctx.store = store
        ctx.solve = res
        ctx.adjoint_rtol = adjoint_rtol
        ctx.max_iters = max_iters
        ctx.solver = solver
        ctx.save_for_backward(alpha)
        return alpha

    @staticmethod
    def backward(ctx, grad_alpha):
        (alpha,) = ctx.saved_tensors
        dimage, dgamma, _, res = ctx.store.adjoint(alpha, grad_alpha.detach().to(torch.float32).contiguous(),
                                                   solver=ctx.solver, rtol=ctx.adjoint_rtol, max_iters=ctx.max_iters)
        ctx.adjoint_solve = res
        return dimage[..., :3].contiguous(), dgamma, None, None, None, None, None, None, None


def levin_matte(image, gamma, s, eps: float = 1e-5, precision: str = "fp16", rtol: float = 1e-6,
                max_iters: int = 5000, adjoint_rtol: float | None = None, solver: str = "mg"):
    """Differentiable matte: alpha (H, W) from image (H, W, 3) in [0, 1],
    per-pixel scribble weights gamma and targets s (both (H, W)).  solver:
    "mg" (multigrid-preconditioned CG, the default: the fastest solve, and the
    one whose adjoint converges at every size and eps tried), "cg" or "pcg"
    (Jacobi-preconditioned) for both the solve and the adjoint; an adjoint
    solve with "cg" or "pcg" that does not converge is redone with "mg"."""
    return LevinMatte.apply(image, gamma, s, eps, precision, rtol, max_iters,
                            rtol if adjoint_rtol is None else adjoint_rtol, solver)
