"""Timing cases of the sparse-GP layer path, through the entry points a program calls.

Each case is one call (or one forward + backward) of ``geepee_gb300.kernels``,
``geepee_gb300.autograd``, ``geepee_gb300.serving`` or ``geepee_gb300.aep_models`` on inputs of
the sizes and distributions of this repository's workloads: the 1-D regression (N = 1000,
M = 30), the psi statistics (N = 10000, Q = 5, M = 100), the 2-layer deep GP (N = 20000, D = 8,
hidden width 2, M = 100, minibatch 1000), the state-space model (M = 50, two states, four
outputs) and the serving mix (M of 50, 100, 200, batches of 1 to 4096 rows).  ``exact`` is
the same quantity in plain float64 torch.
"""
import math

import numpy as np
import torch

from geepee_gb300 import aep_models, autograd, kernels, serving

F64 = torch.float64
JITTER = 1e-5   # on the diagonal of every Kuu
ALPHA = 0.5     # the power of every objective here


def listed():
    return [
        # the smallest call: one uncertain point against a handful of pseudo-inputs, as a
        # controller or a plotting loop asks for; launches and host time only
        dict(name='psi_point', op='weave', n=1, m=24, q=2),
        # the reference's weave loop at the deep GP's second layer: per-point psi2 written out
        dict(name='psi_weave_dgp', op='weave', n=1000, m=100, q=2),
        # gradients for an arbitrary per-point upstream dL/dpsi2, odd sizes (a user's own bound)
        dict(name='psi_deriv_ragged', op='deriv', n=301, m=67, q=3),
        # kernel rows of the whole training set (prediction features, Kuf)
        dict(name='kernel_rows', op='kern', n=20000, m=100, q=8),
        # the deep GP's second layer on a minibatch, forward and backward
        dict(name='layer_dgp', op='psi', n=1000, m=100, q=2, d=1, dtype='float64'),
        # the state-space model's transition over its whole series, two outputs, odd length
        dict(name='layer_ssm', op='psi', n=4999, m=50, q=2, d=2, dtype='float64'),
        # the psi-statistics workload, in both precisions the entry point takes
        dict(name='layer_psi_f64', op='psi', n=10000, m=100, q=5, d=1, dtype='float64'),
        dict(name='layer_psi_f32', op='psi', n=10000, m=100, q=5, d=1, dtype='float32'),
        # the deep GP's first layer over the whole training set, forward and backward
        dict(name='layer_det', op='det', n=20000, m=100, q=8, d=2, dtype='float64'),
        # a served prediction of the largest resident model, an odd batch of rows
        dict(name='serve_m200', op='serve', n=777, m=200, q=8),
        # a long forecast of the state-space model: one step after the other
        dict(name='forecast', op='forecast', n=1000, m=50, q=2),
        # one training step of the deep GP: energy and gradients from host arrays to host arrays
        dict(name='dgp_step', op='dgp', n=20000, m=100, q=8, mb=1000),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(['weave', 'deriv', 'kern', 'psi', 'psi', 'psi', 'det', 'serve', 'forecast', 'dgp'])
    if op == 'weave':
        m = _log_int(rng, 5, 128)
        return dict(op=op, n=_log_int(rng, 1, min(4000, 20000000 // (m * m))), m=m, q=rng.randint(1, 8))
    if op == 'deriv':
        return dict(op=op, n=_log_int(rng, 1, 1000), m=_log_int(rng, 5, 100), q=rng.randint(1, 8))
    if op == 'kern':
        return dict(op=op, n=_log_int(rng, 1, 20000), m=_log_int(rng, 5, 200), q=rng.randint(1, 16))
    if op == 'psi':
        return dict(op=op, n=_log_int(rng, 1, 10000), m=_log_int(rng, 5, 100), q=rng.randint(1, 5), d=rng.randint(1, 2),
                    dtype=rng.choice(['float64', 'float64', 'float32']))
    if op == 'det':
        return dict(op=op, n=_log_int(rng, 1, 20000), m=_log_int(rng, 5, 200), q=rng.randint(1, 16), d=rng.randint(1, 4),
                    dtype=rng.choice(['float64', 'float64', 'float32']))
    if op == 'serve':
        return dict(op=op, n=_log_int(rng, 1, 1024), m=rng.choice([50, 100, 200]), q=8)
    if op == 'forecast':
        return dict(op=op, n=_log_int(rng, 10, 1000), m=_log_int(rng, 10, 100), q=rng.randint(1, 3))
    return dict(op=op, n=_log_int(rng, 3000, 20000), m=_log_int(rng, 20, 100), q=8, mb=_log_int(rng, 50, 2000))


# ------------------------------------------------------------------------------------------
# inputs (host float64, from the seed alone)
# ------------------------------------------------------------------------------------------
def _psi_inputs(case, rng):
    """Input moments, pseudo-inputs and hyperparameters of the psi-statistics workload."""
    N, M, Q = case['n'], case['m'], case['q']
    return dict(mu=rng.randn(N, Q), S=np.exp(rng.uniform(math.log(1e-3), 0.0, (N, Q))), Z=rng.randn(M, Q),
                lls2=2.0 * rng.uniform(-0.5, 0.5, Q), lsf2=2.0 * rng.uniform(-0.2, 0.2, 1))


def _det_inputs(case, rng):
    """Inputs ~ N(0, I); lengthscales as the initialiser sets them (half the typical distance)."""
    N, M, Q = case['n'], case['m'], case['q']
    return dict(x=rng.randn(N, Q), Z=rng.randn(M, Q), lls2=math.log(Q / 2.0) + 2.0 * rng.uniform(-0.2, 0.2, Q),
                lsf2=2.0 * rng.uniform(-0.2, 0.2, 1))


def _layer_weights(M, D, rng):
    """A and a symmetric B of a layer, and upstream gradients are drawn beside them."""
    B = rng.randn(D, M, M) / M
    return rng.randn(D, M) / M, 0.5 * (B + B.transpose(0, 2, 1))


def _q_natural(M, D, rng, suffix):
    """q(u) as the initialiser draws it: mean linspace(-1, 1), covariance factors diag(U(0, 1/2))."""
    iu = np.triu_indices(M)
    e1, e2 = np.zeros((D, len(iu[0]))), np.zeros((D, M))
    for d in range(D):
        a = 0.5 * rng.uniform(0.05, 1.0, M)
        R = np.diag(0.5 * np.log(1.0 / a))
        e1[d], e2[d] = R[iu], np.linspace(-1, 1, M) / a
    return {'eta1_R' + suffix: e1, 'eta2' + suffix: e2}


def _grid_points(M, Q, rng):
    """M pseudo-inputs spread over [-2, 2]^Q (trained pseudo-inputs keep apart)."""
    if Q == 1:
        return np.linspace(-2, 2, M)[:, None] + 0.1 * rng.uniform(-2.0 / M, 2.0 / M, (M, 1))
    side = int(math.ceil(M ** (1.0 / Q)))
    g = np.stack(np.meshgrid(*[np.linspace(-2, 2, side)] * Q, indexing='ij'), -1).reshape(-1, Q)
    return g[rng.permutation(len(g))[:M]] + 0.1 * rng.uniform(-2.0 / side, 2.0 / side, (M, Q))


def _spread_ls(M, Q):
    """Log-lengthscales of such a layer: one spacing of its pseudo-inputs."""
    side = M if Q == 1 else int(math.ceil(M ** (1.0 / Q)))
    return np.full(Q, math.log(max(4.0 / max(side - 1, 1), 0.05)))


def _dgp_params(case, rng, x):
    """Parameters of a 2-layer deep GP (hidden width 2, one output)."""
    M, D = case['m'], case['q']
    p = {'ls_0': np.log(0.5 * math.sqrt(2.0 * D)) + 0.1 * rng.randn(D), 'sf_0': np.log(np.array([0.5])) + 0.05,
         'zu_0': x[rng.permutation(x.shape[0])[:M]].copy()}
    p.update(_q_natural(M, 2, rng, '_0'))
    p.update({'ls_1': _spread_ls(M, 2), 'sf_1': np.zeros(1), 'zu_1': _grid_points(M, 2, rng)})
    p.update(_q_natural(M, 1, rng, '_1'))
    p['sn'] = np.array(math.log(0.1))
    return p


def _dgp_data(case, rng):
    """x ~ N(0, I_D), y = tanh(W2 sin(W1 x)) + N(0, 0.05^2) with hidden width 2."""
    N, D = case['n'], case['q']
    x = rng.randn(N, D)
    W1, W2 = rng.randn(2, D), rng.randn(1, 2)
    return x, np.tanh(np.sin(x @ W1.T) @ W2.T) + 0.05 * rng.randn(N, 1)


def _ssm_params(case, rng):
    """A state-space model's data (four outputs) and parameters; its states of variance 0.1."""
    T, M, Q = 200, case['m'], case['q']
    x = np.cumsum(0.3 * rng.randn(T, Q), 0)
    x = 2.0 * np.sin(x)
    C = rng.randn(4, Q)
    y = x @ C.T + 0.1 * rng.randn(T, 4)
    p = {'sn': math.log(0.05) * np.ones(1), 'x_factor_1': (x / 0.1) / 3, 'x_factor_2': np.log((1 / 0.1) / 3) / 2 * np.ones((T, Q)),
         'C_emission': C + 0.05 * rng.randn(4, Q), 'R_emission': math.log(0.1) * np.ones(4),
         'ls_dynamic': _spread_ls(M, Q) + 0.2, 'sf_dynamic': np.zeros(1), 'zu_dynamic': _grid_points(M, Q, rng)}
    p.update(_q_natural(M, Q, rng, '_dynamic'))
    return y, p


def _inputs(case, seed):
    rng = np.random.RandomState(seed)
    op = case['op']
    if op in ('weave', 'deriv', 'psi'):
        t = _psi_inputs(case, rng)
        if op == 'deriv':
            t['d1'] = rng.randn(case['n'], case['m'])
            d2 = rng.randn(case['n'], case['m'], case['m']) / case['m']
            t['d2'] = 0.5 * (d2 + d2.transpose(0, 2, 1))
    elif op in ('kern', 'det'):
        t = _det_inputs(case, rng)
    if op in ('psi', 'det'):
        t['A'], t['B'] = _layer_weights(case['m'], case['d'], rng)
        t['dm'], t['dv'] = rng.randn(case['n'], case['d']), rng.randn(case['n'], case['d'])
    if op in ('dgp', 'serve'):
        x, y = _dgp_data(case, rng)
        xz = x if op == 'dgp' else rng.randn(2000, case['q'])
        t = dict(x=x, y=y, params=_dgp_params(case, rng, xz), rng_seed=int(rng.randint(1 << 30)))
    if op == 'forecast':
        y, p = _ssm_params(case, rng)
        t = dict(y=y, params=p)
    return t


def prepare(case, seed):
    t, op = _inputs(case, seed), case['op']
    dtype = getattr(torch, case.get('dtype', 'float64'))
    put = lambda a: torch.as_tensor(a, dtype=F64).to('cuda').to(dtype).contiguous()
    if op in ('weave', 'deriv', 'kern'):
        s = {k: put(v) for k, v in t.items()}
        if op == 'deriv':   # lengthscales and variance, and psi as the forward call left it
            s['ell'], s['sf2'] = torch.exp(0.5 * s['lls2']), torch.exp(s['lsf2'])
            s['psi1'], s['psi2'] = kernels.compute_psi_weave(s['lls2'], s['lsf2'], s['mu'], s['S'], s['Z'])
    elif op in ('psi', 'det'):
        s = {k: put(v) for k, v in t.items()}
        for k in ('mu', 'S', 'x', 'Z', 'lls2', 'lsf2', 'A', 'B'):
            if k in s:
                s[k].requires_grad_(True)
    elif op == 'serve':
        M = case['m']
        s = dict(model=serving.ResidentDGP(t['params'], [case['q'], 2, 1], [M, M], torch.device('cuda', 0)), x=put(t['x']))
    elif op == 'forecast':
        s = dict(model=aep_models.SGPSSM(t['y'], case['q'], case['m']))
        s['model'].update_hypers(t['params'])
    else:
        np.random.seed(t['rng_seed'])
        s = dict(model=aep_models.SDGPR(t['x'], t['y'], case['m'], [2]), params=t['params'], rng=np.random.get_state())
        # a training program has the step's graphs captured before its loop begins
        s['model'].objective_function(s['params'], case['mb'], alpha=ALPHA)
    return dict(s, op=op, case=case)


def run(state):
    s, op = state, state['op']
    if op == 'weave':
        return kernels.compute_psi_weave(s['lls2'], s['lsf2'], s['mu'], s['S'], s['Z'])
    if op == 'deriv':
        return kernels.compute_psi_derivatives(s['d1'], s['psi1'], s['d2'], s['psi2'], s['ell'], s['sf2'], s['mu'], s['S'], s['Z'])
    if op == 'kern':
        return kernels.compute_kernel(s['lls2'], s['lsf2'], s['x'], s['Z'])
    if op in ('psi', 'det'):
        if op == 'psi':
            ins = [s[k] for k in ('mu', 'S', 'Z', 'lls2', 'lsf2', 'A', 'B')]
            m, v = autograd.psi_moments(*ins)
        else:
            ins = [s[k] for k in ('x', 'Z', 'lls2', 'lsf2', 'A', 'B')]
            m, v = autograd.det_moments(*ins)
        return (m, v) + torch.autograd.grad((m, v), ins, (s['dm'], s['dv']))
    if op == 'serve':
        return s['model'].predict_y(s['x'])
    if op == 'forecast':
        return s['model'].predict_forward(s['case']['n'])
    np.random.set_state(s['rng'])   # a seeded program: each step's minibatch is reproducible
    energy, grads = s['model'].objective_function(s['params'], s['case']['mb'], alpha=ALPHA)
    return dict(energy=energy, grads=grads)


def work(case):
    """Compulsory bytes (inputs once, outputs once) and operations: an exponential counts as one."""
    op, n, m, q = case['op'], case['n'], case['m'], case['q']
    e = 4 if case.get('dtype') == 'float32' else 8
    pairs = m * (m + 1) // 2
    if op == 'weave':
        return dict(bytes=e * (2 * n * q + m * q + n * m + n * m * m), flops=n * (pairs * (2 * q + 4) + m * 6 * q))
    if op == 'deriv':
        return dict(bytes=e * (4 * n * q + 2 * m * q + n * m + n * m * m), flops=n * (pairs * (2 * q + 5) + m * m * 2 * (q + 1)))
    if op == 'kern':
        return dict(bytes=e * (n * q + m * q + n * m), flops=n * m * (3 * q + 2))
    if op == 'psi':
        d = case['d']
        fwd, bwd = pairs * (2 * q + 4 + 2 * d), pairs * (2 * q + 5 + 4 * d) + m * m * 2 * (q + 1)
        return dict(bytes=e * (4 * n * q + 6 * n * d + 2 * m * q + 2 * d * m * (m + 1)), flops=n * (fwd + bwd))
    if op == 'det':
        d = case['d']
        return dict(bytes=e * (2 * n * q + 6 * n * d + 2 * m * q + 2 * d * m * (m + 1)),
                    flops=n * (m * (3 * q + 2) + d * m * m * 2 + d * m * m + m * (6 * d + 5 * q)))
    if op == 'serve':
        return dict(bytes=e * (n * q + 2 * n + m * (q + 2) + 3 * m * m + 3 * m), flops=n * (m * (3 * q + 2) + 4 * m * m + pairs * 10))
    if op == 'forecast':
        return dict(bytes=e * (m * q + q * m * m + n * 2 * (q + 8)), flops=n * pairs * (2 * q + 4 + 2 * q))
    mb = case['mb']
    host = 2 * (3 * (m * (m + 1) // 2 + m) + m * (q + 2) + q + 5)
    algebra = 3 * m ** 3 * 30   # two factorisations and about thirty M x M products of three outputs
    rows = mb * (m * (3 * q + 2) + 6 * m * m + m * (12 + 5 * q) + pairs * 28 + m * m * 6)
    return dict(bytes=8 * (host + mb * (q + 1)), flops=algebra + rows)


# ------------------------------------------------------------------------------------------
# the same quantities in plain float64 torch
# ------------------------------------------------------------------------------------------
def _psi_stats(mu, S, Z, lls2, lsf2):
    """psi1 [n, M] and psi2 [n, M, M] of the ARD exponentiated-quadratic kernel under N(mu, S)."""
    l = torch.exp(lls2)
    d1 = l + S
    e1 = (0.5 * torch.log(l / d1)[:, None, :] - 0.5 * (mu[:, None, :] - Z[None]) ** 2 / d1[:, None, :]).sum(-1)
    d2 = l + 2.0 * S
    zbar = 0.5 * (Z[:, None, :] + Z[None])
    zz = ((Z[:, None, :] - Z[None]) ** 2 / (4.0 * l)).sum(-1)
    e2 = (0.5 * torch.log(l / d2)).sum(-1)[:, None, None] - zz
    for q in range(Z.shape[1]):
        e2 = e2 - (mu[:, q, None, None] - zbar[None, :, :, q]) ** 2 / d2[:, q, None, None]
    return torch.exp(lsf2 + e1), torch.exp(2.0 * lsf2 + e2)


def _kernel(x, Z, lls2, lsf2):
    e = x.new_zeros(x.shape[0], Z.shape[0])
    for q in range(Z.shape[1]):
        e = e - 0.5 * (x[:, q, None] - Z[None, :, q]) ** 2 / torch.exp(lls2[q])
    return torch.exp(lsf2 + e)


def _psi_layer(mu, S, Z, lls2, lsf2, A, B):
    p1, p2 = _psi_stats(mu, S, Z, lls2, lsf2)
    m = p1 @ A.T
    return m, torch.exp(lsf2) + p2.reshape(p2.shape[0], -1) @ B.reshape(B.shape[0], -1).T - m * m


def _det_layer(x, Z, lls2, lsf2, A, B):
    k = _kernel(x, Z, lls2, lsf2)
    v = torch.stack([((k @ B[d]) * k).sum(-1) for d in range(B.shape[0])], 1)
    return k @ A.T, torch.exp(lsf2) + v


def _grads_by_chunks(layer, rows, shared, dm, dv, step):
    """Outputs and gradients of sum(dm m + dv v), `step` rows at a time."""
    shared = [t.clone().requires_grad_(True) for t in shared]
    ms, vs, gr = [], [], [[] for _ in rows]
    gs = [torch.zeros_like(t) for t in shared]
    for a in range(0, dm.shape[0], step):
        r = [t[a:a + step].clone().requires_grad_(True) for t in rows]
        m, v = layer(*r, *shared)
        g = torch.autograd.grad((dm[a:a + step] * m).sum() + (dv[a:a + step] * v).sum(), r + shared)
        for i in range(len(rows)):
            gr[i].append(g[i])
        for i in range(len(shared)):
            gs[i] += g[len(rows) + i]
        ms.append(m.detach())
        vs.append(v.detach())
    return [torch.cat(ms), torch.cat(vs)] + [torch.cat(g) for g in gr] + gs


def _gp_layer(p, sfx, beta):
    """Moments of q(u) with its natural parameters scaled by beta (1: the posterior): A, B for
    deterministic inputs, and log det(I + K T), mean . theta_2 for the log-partition.  With
    T = beta theta_1, t = beta theta_2: B = -(I + T K)^-1 T, A = (I + T K)^-1 t, mean = K A."""
    Z, lls2, lsf2 = p['zu' + sfx], 2.0 * p['ls' + sfx], 2.0 * p['sf' + sfx]
    M = Z.shape[0]
    K = _kernel(Z, Z, lls2, lsf2) + JITTER * torch.eye(M, dtype=F64, device=Z.device)
    iu = torch.triu_indices(M, M, device=Z.device)
    D = p['eta2' + sfx].shape[0]
    R = torch.zeros(D, M, M, dtype=F64, device=Z.device)
    R = R.index_put((torch.arange(D, device=Z.device)[:, None], iu[0][None], iu[1][None]), p['eta1_R' + sfx])
    dg = torch.diagonal(R, dim1=1, dim2=2)
    R = R - torch.diag_embed(dg) + torch.diag_embed(torch.exp(dg))
    T = beta * R.transpose(1, 2) @ R
    ITK = torch.eye(M, dtype=F64, device=Z.device) + T @ K
    B = -torch.linalg.solve(ITK, T)
    A = torch.linalg.solve(ITK, beta * p['eta2' + sfx].unsqueeze(-1)).squeeze(-1)
    quad = ((A @ K) * p['eta2' + sfx]).sum() * beta
    return A, 0.5 * (B + B.transpose(1, 2)), torch.linalg.slogdet(ITK)[1].sum(), quad


def _predict(p, x):
    A, B, _, _ = _gp_layer(p, '_0', 1.0)
    m, v = _det_layer(x, p['zu_0'], 2.0 * p['ls_0'], 2.0 * p['sf_0'], A, B)
    A, B, _, _ = _gp_layer(p, '_1', 1.0)
    m, v = _psi_layer(m, v, p['zu_1'], 2.0 * p['ls_1'], 2.0 * p['sf_1'], A, B + A[:, :, None] * A[:, None, :])
    return m, v + torch.exp(2.0 * p['sn'])


def _dgp_energy(p, x, y, N, alpha):
    """The energy of the 2-layer deep GP (Gaussian likelihood) on minibatch rows x, y."""
    beta = (N - alpha) / N
    phi, hid = 0.0, []
    for sfx in ('_0', '_1'):
        _, _, ld, quad = _gp_layer(p, sfx, 1.0)
        A, B, ldh, quadh = _gp_layer(p, sfx, beta)
        phi = phi + (N / alpha - 1.0) * 0.5 * (quad - ld) - (N / alpha) * 0.5 * (quadh - ldh)
        hid.append((A, B))
    (A0, B0), (A1, B1) = hid
    m, v = _det_layer(x, p['zu_0'], 2.0 * p['ls_0'], 2.0 * p['sf_0'], A0, B0)
    m, v = _psi_layer(m, v, p['zu_1'], 2.0 * p['ls_1'], 2.0 * p['sf_1'], A1, B1 + A1[:, :, None] * A1[:, None, :])
    sn2 = torch.exp(2.0 * p['sn'])
    vt, r, nb = v + sn2 / alpha, y - m, y.shape[0]
    logZ = (-0.5 * (torch.log(2 * math.pi * vt) + r * r / vt)).sum()
    logZ = logZ + nb * (0.5 * torch.log(2 * math.pi * sn2 / alpha) - 0.5 * alpha * torch.log(2 * math.pi * sn2))
    return (-N / nb / alpha * logZ + phi).sum() / N


def exact(case, seed):
    t, op = _inputs(case, seed), case['op']
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    dtype = getattr(torch, case.get('dtype', 'float64'))
    put = lambda a: torch.as_tensor(a, dtype=F64).to(dev).to(dtype).to(F64)   # the values that run() is given
    step = max(1, 10000000 // (case['m'] * case['m']))
    if op == 'kern':
        return _kernel(*[put(t[k]) for k in ('x', 'Z', 'lls2', 'lsf2')])
    if op == 'weave':
        return _psi_stats(*[put(t[k]) for k in ('mu', 'S', 'Z', 'lls2', 'lsf2')])
    if op == 'deriv':
        mu, S, Z, lls2, lsf2, d1, d2 = [put(t[k]) for k in ('mu', 'S', 'Z', 'lls2', 'lsf2', 'd1', 'd2')]
        ell, sf2 = torch.exp(0.5 * lls2), torch.exp(lsf2)
        v = [w.requires_grad_(True) for w in (sf2, ell, Z, mu, S)]
        p1, p2 = _psi_stats(mu, S, Z, 2.0 * torch.log(ell), torch.log(sf2))
        g = torch.autograd.grad((d1 * p1).sum() + (d2 * p2).sum(), v)
        return (g[0][0],) + tuple(g[1:])
    if op == 'psi':
        rows, shared = [put(t[k]) for k in ('mu', 'S')], [put(t[k]) for k in ('Z', 'lls2', 'lsf2', 'A', 'B')]
        return _grads_by_chunks(_psi_layer, rows, shared, put(t['dm']), put(t['dv']), step)
    if op == 'det':
        rows, shared = [put(t['x'])], [put(t[k]) for k in ('Z', 'lls2', 'lsf2', 'A', 'B')]
        return _grads_by_chunks(_det_layer, rows, shared, put(t['dm']), put(t['dv']), 20000)
    p = {k: put(np.asarray(v)) for k, v in t['params'].items()}
    if op == 'serve':
        return _predict(p, put(t['x']))
    if op == 'forecast':
        A, B, _, _ = _gp_layer(p, '_dynamic', 1.0)
        Bs = B + A[:, :, None] * A[:, None, :]
        f1, f2 = p['x_factor_1'][-1:], torch.exp(2.0 * p['x_factor_2'][-1:])
        m, v, ms, vs = f1 / f2, 0.5 / f2, [], []   # two factors reach the last state
        for _ in range(case['n']):
            m, v = _psi_layer(m, v, p['zu_dynamic'], 2.0 * p['ls_dynamic'], 2.0 * p['sf_dynamic'], A, Bs)
            ms.append(m)
            vs.append(v)
        mx, vx = torch.cat(ms), torch.cat(vs)
        C, R = p['C_emission'], torch.exp(2.0 * p['R_emission'])
        vyn = vx @ (C * C).T
        return mx, vx, mx @ C.T, vyn, vyn + R
    np.random.seed(t['rng_seed'])
    idx = np.random.choice(case['n'], case['mb'], replace=False)
    p = {k: w.requires_grad_(True) for k, w in p.items()}
    e = _dgp_energy(p, put(t['x'][idx]), put(t['y'][idx]), case['n'], ALPHA)
    g = torch.autograd.grad(e, list(p.values()))
    return dict(energy=e.item(), grads={k: w.reshape(np.shape(t['params'][k])) for k, w in zip(p, g)})
