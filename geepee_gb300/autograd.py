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


class _Sums:
    """One backward call's float64 sums, [dsf2 | dl | dZ | dA | dB], with the two chained
    hyperparameter gradients behind them, and for float32 layers the casts of dZ, dA, dB."""

    def __init__(self, Q, M, D, dtype, device):
        self.sizes = [1 + Q, M * Q, D * M, D * M * M]
        n = sum(self.sizes)
        self.shapes = ((M, Q), (D, M), (D, M, M))
        buf = torch.empty(n + Q + 1, dtype=torch.float64, device=device)
        self.acc, self.g_l, self.g_s = buf.split([n, Q, 1])
        self.cast = None if dtype == torch.float64 else torch.empty(n - 1 - Q, dtype=dtype, device=device)

    def grads(self, hyp):
        """(dZ, g_lls2, g_lsf2, dA, dB) in the inputs' types."""
        (lt, lshape), (st, sshape) = hyp
        rest = self.acc.split(self.sizes)[1:] if self.cast is None else self.cast.split(self.sizes[1:])
        dZ, dA, dB = [t.view(s) for t, s in zip(rest, self.shapes)]
        return dZ, self.g_l.reshape(lshape).to(lt), self.g_s.reshape(sshape).to(st), dA, dB


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
        sums = _Sums(Q, M, D, mu.dtype, mu.device)
        dmu, dS = torch.empty_like(mu), torch.empty_like(S)
        work = torch.empty(gpk.work_elems(gpk.OP_PSI_BWD, N, M, Q, D), dtype=torch.float64, device=mu.device)
        gpk.psi_layer_bwd(mu, S, Z, l2, s2, A, B, m, dm, dv, sums.acc, dmu, dS, sums.g_l, sums.g_s, sums.cast, work)
        dZ, g_l, g_s, dA, dB = sums.grads(ctx.hyp)
        return dmu, dS, dZ, g_l, g_s, dA, dB


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
        sums = _Sums(Q, M, D, x.dtype, x.device)
        dx = torch.empty_like(x)
        n1, n2 = gpk.work_elems(gpk.OP_DET_BWD, N, M, Q, D), gpk.work_elems(gpk.OP_GRAM, N, M, Q, D)
        work = torch.empty(max(n1, n2), dtype=torch.float64, device=x.device)   # one after the other
        gpk.det_layer_bwd(x, Z, l2, s2, A, kfu, Bk, dm, dv, sums.acc, dx, sums.g_l, sums.g_s, sums.cast, work)
        dZ, g_l, g_s, dA, dB = sums.grads(ctx.hyp)
        return dx, dZ, g_l, g_s, dA, dB


def psi_moments(mu, S, Z, lls2, lsf2, A, B):
    """Differentiable (m, v) of a sparse-GP layer under Gaussian inputs; see the module docstring."""
    return PsiMoments.apply(mu, S, Z, lls2, lsf2, A, B)


def det_moments(x, Z, lls2, lsf2, A, B):
    """Differentiable (m, v) of a sparse-GP layer under deterministic inputs."""
    return DetMoments.apply(x, Z, lls2, lsf2, A, B)
