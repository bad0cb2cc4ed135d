"""torch.autograd.Function over the libgmgs adjoint (extension beyond the
reference, which has no density field and no gradients).

    J = compliance(rho, solver)                 # F^T U(rho)
    J = displacement_functional(rho, solver, ell)   # ell^T U(rho)
    J.backward()                                # rho.grad = dJ/drho from gmgs_grad

The forward pass sets the per-voxel stiffness scale rho^penal on the finest
level (gmgs_set_density), solves with the handle's PCG and returns J; the
backward pass calls gmgs_grad, which for compliance uses U itself and for a
displacement functional solves the adjoint system K lambda = ell with the same
PCG, then reduces -penal rho^(penal-1) lambda_e^T Ke0 u_e per voxel on the GPU.
The handle keeps the state of the last forward pass, so call backward before
the next forward on the same solver.
"""
from __future__ import annotations

import numpy as np
import torch

from .solver import Solver


def _on_handle_device(t: torch.Tensor) -> bool:
    """Whether t lives where the library's calls run: the current CUDA device."""
    return t.is_cuda and t.device.index == torch.cuda.current_device()


class _Functional(torch.autograd.Function):
    # Densities and gradients of a CUDA tensor stay on the device, and the
    # compliance is one dot product there: a round trip of the densities, U and
    # the gradient through host memory took as long as the solve of an 84 x 73
    # x 128 model.  The library works on the handle's stream, so torch's current
    # stream is waited for before it touches a tensor of torch's allocator.
    @staticmethod
    def forward(ctx, rho: torch.Tensor, solver: Solver, penal: float, ell):
        r = rho.detach()
        if _on_handle_device(r):
            if r.numel() != solver.num_elements(1):
                raise ValueError("rho must have one entry per solid voxel")
            r = r.to(torch.float64).contiguous()
            torch.cuda.current_stream().synchronize()
            solver.set_density_dev(r.data_ptr(), penal)
        else:
            solver.set_density(r.to("cpu", torch.float64).numpy().ravel(), penal)
        if ell is None:
            solver.solve_dev(None)
            J = solver.load_work()
        else:
            J = float(np.asarray(ell, dtype=np.float64).ravel() @ solver.solve())
        ctx.solver = solver
        ctx.ell = ell
        ctx.rho_meta = (rho.shape, rho.dtype, rho.device)
        return torch.tensor(J, dtype=rho.dtype, device=rho.device)

    @staticmethod
    def backward(ctx, gout):
        shape, dtype, device = ctx.rho_meta
        if ctx.ell is None and device.type == "cuda" and device.index == torch.cuda.current_device():
            g = torch.empty(ctx.solver.num_elements(1), dtype=torch.float64, device=device)
            torch.cuda.current_stream().synchronize()
            ctx.solver.grad_dev(None, g.data_ptr())
            grad = g.to(dtype)
        else:
            grad = torch.as_tensor(ctx.solver.grad(ctx.ell), dtype=dtype, device=device)
        return grad.reshape(shape) * gout, None, None, None


def compliance(rho: torch.Tensor, solver: Solver, penal: float = 3.0) -> torch.Tensor:
    """F^T U for the stiffness scale rho^penal (one entry per solid voxel)."""
    return _Functional.apply(rho, solver, penal, None)


def displacement_functional(rho: torch.Tensor, solver: Solver, ell, penal: float = 3.0) -> torch.Tensor:
    """ell^T U; ell is a 3*num_nodes interleaved vector (e.g. one tip DOF)."""
    return _Functional.apply(rho, solver, penal, ell)
