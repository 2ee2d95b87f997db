"""torch.autograd.Function wrappers of the layer kernels, so that torch code can differentiate
through the psi statistics and the deterministic layer with the hand-written backward kernels.

* ``psi_moments(mu, S, Z, lls2, lsf2, A, B)`` -> (m, v): a sparse-GP layer's output moments under
  Gaussian inputs N(mu, S) (geepee/aep_models.py:182-199 with compute_psi_weave,
  kernels.py:181-240): m = psi1 A^T, v = sf2 + sum_ab B[d] psi2[n] - m^2.  Forward gpk_psi_fwd;
  backward gpk_psi_bwd, which recomputes psi1 and psi2 (nothing N x M x M is stored) - the role
  of compute_psi_derivatives (kernels.py:302-309) in backprop_grads_lvm_mm
  (aep_models.py:201-304).
* ``det_moments(x, Z, lls2, lsf2, A, B)`` -> (m, v): the same layer under deterministic inputs
  (aep_models.py:142-158): m = Kfu A^T, v = sf2 + rowdiag(Kfu B Kfu^T), B symmetric (as Bhat
  is).  Forward gpk_det_fwd; backward gpk_det_bwd (compute_kfu_derivatives, kernels.py:312-313)
  and gpk_gram for dB.

Hyperparameters are in the reference's log form: lls2 [Q] = log ell^2, lsf2 [1] = log sf^2.
Tensors are CUDA float64 (double-float arithmetic) or float32; the sums over points reach the
gradients in a fixed order, so repeated backward passes give identical results.
"""
from __future__ import annotations

import torch

from . import gpk

__all__ = ['PsiMoments', 'DetMoments', 'psi_moments', 'det_moments']


def _c(t):
    return t.detach().contiguous()


def _hyp(lls2, lsf2):
    """The hyperparameters as the kernels take them: contiguous float64."""
    return _c(lls2).double(), _c(lsf2).double().reshape(1)


def _up(g, like):
    """An upstream gradient (None: zero) as a contiguous tensor of the outputs' type."""
    return torch.zeros_like(like) if g is None else g.contiguous().to(like.dtype)


def _shared_grads(Z, A, hyp):
    """Gradients of what all rows share, uninitialised, each a tensor of its own: (dZ, dA, dB) in the
    layer's type, (g_lls2, g_lsf2) in float64 and the hyperparameters' shapes; and the number of
    float64 sums that the backward keeps beside them (float32 layers sum in float64 first)."""
    (M, Q), D = Z.shape, A.shape[0]
    dZ, dA = torch.empty_like(Z), torch.empty_like(A)
    dB = torch.empty((D, M, M), dtype=A.dtype, device=A.device)
    g_l, g_s = [torch.empty(shape, dtype=torch.float64, device=Z.device) for _, shape in hyp]
    return dZ, dA, dB, g_l, g_s, 1 + Q + (0 if Z.dtype == torch.float64 else M * Q + D * M + D * M * M)


def _hyp_kind(lls2, lsf2):
    return ((lls2.dtype, lls2.shape), (lsf2.dtype, lsf2.shape))


class PsiMoments(torch.autograd.Function):
    @staticmethod
    def forward(ctx, mu, S, Z, lls2, lsf2, A, B):
        mu, S, Z, A, B = _c(mu), _c(S), _c(Z), _c(A), _c(B)
        l2, s2 = _hyp(lls2, lsf2)
        m = torch.empty((mu.shape[0], A.shape[0]), dtype=mu.dtype, device=mu.device)
        v = torch.empty_like(m)
        gpk.psi_fwd(mu, S, Z, l2, s2, A, B, m_out=m, v_out=v)
        ctx.save_for_backward(mu, S, Z, l2, s2, A, B, m)
        ctx.hyp = _hyp_kind(lls2, lsf2)
        return m, v

    @staticmethod
    def backward(ctx, dm, dv):
        mu, S, Z, l2, s2, A, B, m = ctx.saved_tensors
        N, Q = mu.shape
        M, D = Z.shape[0], A.shape[0]
        dm, dv = _up(dm, m), _up(dv, m)
        dZ, dA, dB, g_l, g_s, nsums = _shared_grads(Z, A, ctx.hyp)
        dmu, dS = torch.empty_like(mu), torch.empty_like(S)
        work = torch.empty(nsums + gpk.work_elems(gpk.OP_PSI_BWD, N, M, Q, D), dtype=torch.float64, device=mu.device)
        gpk.psi_layer_bwd(mu, S, Z, l2, s2, A, B, m, dm, dv, dZ, dA, dB, dmu, dS, g_l, g_s, work)
        return dmu, dS, dZ, g_l.to(ctx.hyp[0][0]), g_s.to(ctx.hyp[1][0]), dA, dB


class DetMoments(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, Z, lls2, lsf2, A, B):
        x, Z, A, B = _c(x), _c(Z), _c(A), _c(B)
        l2, s2 = _hyp(lls2, lsf2)
        N, M, D = x.shape[0], Z.shape[0], A.shape[0]
        kfu = torch.empty((N, M), dtype=x.dtype, device=x.device)
        Bk = torch.empty((N, D, M), dtype=x.dtype, device=x.device)
        m = torch.empty((N, D), dtype=x.dtype, device=x.device)
        v = torch.empty_like(m)
        gpk.det_fwd(x, Z, l2, s2, A, B, kfu, Bk, m, v)
        ctx.save_for_backward(x, Z, l2, s2, A, kfu, Bk)
        ctx.hyp = _hyp_kind(lls2, lsf2)
        return m, v

    @staticmethod
    def backward(ctx, dm, dv):
        x, Z, l2, s2, A, kfu, Bk = ctx.saved_tensors
        N, Q = x.shape
        M, D = Z.shape[0], A.shape[0]
        dm = torch.zeros((N, D), dtype=x.dtype, device=x.device) if dm is None else _up(dm, x)
        dv = torch.zeros((N, D), dtype=x.dtype, device=x.device) if dv is None else _up(dv, x)
        dZ, dA, dB, g_l, g_s, nsums = _shared_grads(Z, A, ctx.hyp)
        dx = torch.empty_like(x)
        n1, n2 = gpk.work_elems(gpk.OP_DET_BWD, N, M, Q, D), gpk.work_elems(gpk.OP_GRAM, N, M, Q, D)
        work = torch.empty(nsums + max(n1, n2), dtype=torch.float64, device=x.device)   # one after the other
        gpk.det_layer_bwd(x, Z, l2, s2, A, kfu, Bk, dm, dv, dZ, dA, dB, dx, g_l, g_s, work)
        return dx, dZ, g_l.to(ctx.hyp[0][0]), g_s.to(ctx.hyp[1][0]), dA, dB


def psi_moments(mu, S, Z, lls2, lsf2, A, B):
    """Differentiable (m, v) of a sparse-GP layer under Gaussian inputs; see the module docstring."""
    return PsiMoments.apply(mu, S, Z, lls2, lsf2, A, B)


def det_moments(x, Z, lls2, lsf2, A, B):
    """Differentiable (m, v) of a sparse-GP layer under deterministic inputs."""
    return DetMoments.apply(x, Z, lls2, lsf2, A, B)
