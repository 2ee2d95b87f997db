"""The psi statistics at the edges of their kernels' ranges: ragged sizes around the row, pair and
shared-memory limits of the backward's layouts, every input width, and points whose exponents lie
outside the fixed-point range of the double-float pair sweep (they take its general form)."""
import numpy as np
import pytest
import torch

from oracle import geepee_np as O
from tests._helpers import assert_close

pytestmark = pytest.mark.gpu

TOL = 1e-9   # double-float sums (~48 bits) of a few thousand terms against float64


def dev(a, dtype=torch.float64):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device='cuda').to(dtype).contiguous()


def z(*s):
    return torch.zeros(s, dtype=torch.float64, device='cuda')


@pytest.mark.parametrize('M,Q,Dout,N,fixed', [
    (2, 1, 1, 5, True), (13, 2, 3, 9, True), (59, 2, 1, 400, True), (64, 3, 2, 33, True), (65, 4, 1, 35, True),
    (70, 5, 2, 21, False), (104, 2, 1, 170, True), (110, 2, 1, 20, True), (100, 5, 1, 20, True), (96, 6, 1, 11, True),
    (129, 2, 1, 9, True), (129, 7, 1, 5, False), (150, 1, 2, 7, True), (155, 2, 1, 6, False), (31, 8, 4, 40, True)])
def test_psi_layer_edge_sizes(M, Q, Dout, N, fixed):
    """Forward moments and every backward output against the oracle, with the fixed-order sums
    (twice, bit for bit) or the atomic ones."""
    from geepee_gb300 import gpk, workloads as W
    wl = W.psi_workload(seed=3 * M + Q, N=N, Q=Q, M=M, Dout=Dout)
    lls2, lsf2 = 2 * wl['ls'], 2 * wl['sf'] + 0.1
    p1, p2 = O.psi_stats(lls2, lsf2, wl['mu'], wl['S'], wl['Z'])
    A, B, sf2 = wl['Ahat'], wl['Bhat'], float(np.exp(lsf2[0]))
    m_ref = p1 @ A.T
    v_ref = sf2 + np.einsum('dab,nab->nd', B, p2) - m_ref ** 2
    dm, dv = wl['dm'], wl['dv']
    dm_all = dm - 2 * dv * m_ref
    r = O.psi_derivatives(dm_all @ A, p1, np.einsum('nd,dab->nab', dv, B), p2, np.exp(wl['ls']), sf2,
                          wl['mu'], wl['S'], wl['Z'])
    t = {k: dev(wl[k]) for k in ('mu', 'S', 'Z')}
    l2, s2, At, Bt = dev(lls2), dev(lsf2), dev(A), dev(B)
    m, v = z(N, Dout), z(N, Dout)
    gpk.psi_fwd(t['mu'], t['S'], t['Z'], l2, s2, At, Bt, m_out=m, v_out=v)
    assert_close(m.cpu().numpy(), m_ref, TOL, 'm')
    assert_close(v.cpu().numpy(), v_ref, TOL, 'v')
    work = z(gpk.work_elems(gpk.OP_PSI_BWD, N, M, Q, Dout)) if fixed else None
    outs = []
    for _ in range(2):
        out = dict(dsf2=z(1), dl=z(Q), dZ=z(M, Q), dA=z(Dout, M), dB=z(Dout, M, M), dmu=z(N, Q), dS=z(N, Q))
        gpk.psi_bwd(t['mu'], t['S'], t['Z'], l2, s2, At, Bt, dev(m_ref), dev(dm), dev(dv), out['dsf2'], out['dl'],
                    out['dZ'], out['dA'], out['dB'], out['dmu'], out['dS'], work=work)
        outs.append(out)
    for name, val in zip(('dsf2', 'dl', 'dZ', 'dmu', 'dS'), r):
        assert_close(outs[0][name].cpu().numpy(), val, TOL, name)
    assert_close(outs[0]['dA'].cpu().numpy(), dm_all.T @ p1, TOL, 'dA')
    assert_close(outs[0]['dB'].cpu().numpy(), np.einsum('nd,nab->dab', dv, p2), TOL, 'dB')
    if fixed:
        for name in outs[0]:
            assert torch.equal(outs[0][name], outs[1][name]), name + ' differs between calls'


@pytest.mark.parametrize('kind', ['far', 'negative_variance', 'large_sf', 'mixed'])
@pytest.mark.parametrize('Q', [2, 5])
def test_psi_outside_fixed_point_range(kind, Q):
    """Far points (every psi2 zero), slightly negative variances and a kernel variance near the
    float range, alone and beside ordinary points, forward and backward."""
    from geepee_gb300 import gpk, workloads as W
    N, M, Dout = 23, 37, 1
    wl = W.psi_workload(seed=11 + Q, N=N, Q=Q, M=M, Dout=Dout)
    lls2, lsf2 = 2 * wl['ls'], np.array([0.3])
    mu, S = wl['mu'].copy(), wl['S'].copy()
    if kind in ('far', 'mixed'):
        mu[5] = 40.0
        mu[6, 0] = -1e4
        S[6] = 1e-6
        mu[9] *= 8.0
    if kind in ('negative_variance', 'mixed'):
        S[::4] = -0.05 * np.exp(lls2)
        S[7] = 0.0
    if kind == 'large_sf':
        lsf2 = np.array([43.85])   # psi2 up to e^87.7, within the float range; k_n above 126
    p1, p2 = O.psi_stats(lls2, lsf2, mu, S, wl['Z'])
    psi1, psi2 = z(N, M), z(N, M, M)
    t = dict(mu=dev(mu), S=dev(S), Z=dev(wl['Z']))
    l2, s2 = dev(lls2), dev(lsf2)
    gpk.psi_fwd(t['mu'], t['S'], t['Z'], l2, s2, psi1=psi1, psi2=psi2)
    # results below e^-87 may be flushed to zero
    floor = 2e-38
    np.testing.assert_allclose(psi2.cpu().numpy(), p2, rtol=1e-10, atol=floor)
    np.testing.assert_allclose(psi1.cpu().numpy(), p1, rtol=1e-10, atol=floor)
    if kind == 'large_sf':
        return   # sums of such terms leave the float range
    A, B, sf2 = wl['Ahat'], wl['Bhat'], float(np.exp(lsf2[0]))
    m_ref = p1 @ A.T
    m, v = z(N, Dout), z(N, Dout)
    gpk.psi_fwd(t['mu'], t['S'], t['Z'], l2, s2, dev(A), dev(B), m_out=m, v_out=v)
    assert_close(m.cpu().numpy(), m_ref, TOL, 'm')
    assert_close(v.cpu().numpy(), sf2 + np.einsum('dab,nab->nd', B, p2) - m_ref ** 2, TOL, 'v')
    dm, dv = wl['dm'], wl['dv']
    dm_all = dm - 2 * dv * m_ref
    r = O.psi_derivatives(dm_all @ A, p1, np.einsum('nd,dab->nab', dv, B), p2, np.exp(wl['ls']), sf2, mu, S, wl['Z'])
    out = dict(dsf2=z(1), dl=z(Q), dZ=z(M, Q), dA=z(Dout, M), dB=z(Dout, M, M), dmu=z(N, Q), dS=z(N, Q))
    gpk.psi_bwd(t['mu'], t['S'], t['Z'], l2, s2, dev(A), dev(B), dev(m_ref), dev(dm), dev(dv), out['dsf2'],
                out['dl'], out['dZ'], out['dA'], out['dB'], out['dmu'], out['dS'],
                work=z(gpk.work_elems(gpk.OP_PSI_BWD, N, M, Q, Dout)))
    for name, val in zip(('dsf2', 'dl', 'dZ', 'dmu', 'dS'), r):
        assert_close(out[name].cpu().numpy(), val, TOL, name)


def test_psi_nan_stays_with_its_point():
    """A point with a NaN moment gives NaN there and leaves the others of its pass unchanged."""
    from geepee_gb300 import gpk, workloads as W
    N, M, Q = 9, 20, 2
    wl = W.psi_workload(seed=4, N=N, Q=Q, M=M, Dout=1)
    mu = wl['mu'].copy()
    mu[2, 1] = np.nan
    res = []
    for x in (wl['mu'], mu):
        m, v = z(N, 1), z(N, 1)
        gpk.psi_fwd(dev(x), dev(wl['S']), dev(wl['Z']), dev(2 * wl['ls']), dev(2 * wl['sf']), dev(wl['Ahat']),
                    dev(wl['Bhat']), m_out=m, v_out=v)
        res.append((m.cpu().numpy(), v.cpu().numpy()))
    ok = np.arange(N) != 2
    assert np.isnan(res[1][0][2]) and np.isnan(res[1][1][2])
    for a, b in zip(*res):
        assert_close(b[ok], a[ok], 1e-12)


@pytest.mark.parametrize('M,Q', [(1, 1), (3, 2), (50, 2), (51, 2), (49, 3), (100, 4), (110, 1)])
@pytest.mark.parametrize('kind', ['plain', 'far', 'negative_variance'])
def test_psi_rollout_vs_oracle(M, Q, kind):
    """Twelve dependent steps against the oracle's psi statistics; the first from an ordinary state,
    one whose distances underflow every psi2, or one with a slightly negative variance."""
    from geepee_gb300 import gpk
    rng = np.random.RandomState(7 * M + Q)
    Z = rng.uniform(-2, 2, (M, Q))
    lls2, lsf2 = 2 * rng.uniform(-0.6, 0.2, Q), np.array([0.2])
    A = rng.randn(Q, M) / np.sqrt(M)
    B = rng.randn(Q, M, M) / M
    B = 0.1 * (B + B.transpose(0, 2, 1))
    mu, S = rng.randn(Q), np.exp(rng.uniform(-3, 0, Q))
    if kind == 'far':
        mu[0], S = 60.0, 1e-3 * S
    if kind == 'negative_variance':
        S[0] = -0.03 * np.exp(lls2[0])
    T, sf2 = 12, float(np.exp(lsf2[0]))
    ms, vs, m, v = [], [], mu[None], S[None]
    for _ in range(T):
        p1, p2 = O.psi_stats(lls2, lsf2, m, v, Z)
        m = p1 @ A.T
        v = sf2 + np.einsum('dab,nab->nd', B, p2) - m ** 2
        ms.append(m[0])
        vs.append(v[0])
    gm, gv = gpk.psi_rollout(dev(mu), dev(S), dev(Z), dev(lls2), dev(lsf2), dev(A), dev(B), T)
    # (a drawn layer may drive its variance below -l/2, from where on the statistics are NaN)
    ok = int(np.isfinite(np.array(ms)).all(1).cumprod().sum())
    assert_close(gm.cpu().numpy()[:ok], np.array(ms)[:ok], TOL, 'm')
    assert_close(gv.cpu().numpy()[:ok], np.array(vs)[:ok], TOL, 'v')
    assert ok >= 1 and not bool(torch.isfinite(gm[ok:]).all(1).any())
    m1, v1 = gpk.psi_rollout(dev(mu), dev(S), dev(Z), dev(lls2), dev(lsf2), dev(A), dev(B), 1)
    assert torch.equal(m1[0], gm[0]) and torch.equal(v1[0], gv[0])
    bad = mu.copy()
    bad[0] = np.nan
    gm, gv = gpk.psi_rollout(dev(bad), dev(S), dev(Z), dev(lls2), dev(lsf2), dev(A), dev(B), 3)
    assert bool(torch.isnan(gm).all()) and bool(torch.isnan(gv).all())


@pytest.mark.parametrize('N,M,Q,dtype', [(160, 1, 1, 'float64'), (700, 17, 3, 'float64'), (300, 33, 8, 'float64'),
                                         (155, 41, 2, 'float32'), (160, 101, 2, 'float64'), (153, 128, 8, 'float64'),
                                         (153, 128, 8, 'float32'), (153, 140, 5, 'float64')])
def test_psi_points_written_out(N, M, Q, dtype):
    """psi2 of every point at the sizes where the split changes: several small CTAs an SM, two,
    one, and one with a single buffer of pairs.  Same tolerances as the psi statistics'."""
    from geepee_gb300 import gpk
    dt = getattr(torch, dtype)
    rng = np.random.RandomState(N + M)
    Z, mu, S = rng.randn(M, Q), rng.randn(N, Q), rng.uniform(0.01, 1.0, (N, Q))
    lls2, lsf2 = rng.uniform(-0.5, 0.5, Q), np.array([0.3])
    psi1, psi2 = torch.zeros((N, M), dtype=dt, device='cuda'), torch.zeros((N, M, M), dtype=dt, device='cuda')
    gpk.psi_fwd(dev(mu, dt), dev(S, dt), dev(Z, dt), dev(lls2), dev(lsf2), psi1=psi1, psi2=psi2)
    p1, p2 = O.psi_stats(lls2, lsf2, mu, S, Z)
    tol = 1e-10 if dtype == 'float64' else 1e-4
    np.testing.assert_allclose(psi1.cpu().numpy(), p1, rtol=tol, atol=tol * np.abs(p1).max())
    np.testing.assert_allclose(psi2.cpu().numpy(), p2, rtol=tol, atol=tol * np.abs(p2).max())


@pytest.mark.parametrize('M,Q,Dout,N', [(1, 3, 1, 1), (37, 3, 2, 41), (64, 4, 1, 7), (100, 4, 4, 5), (129, 3, 1, 3)])
def test_psi_layer_three_and_four_inputs(M, Q, Dout, N):
    """The width that serves three and four input dimensions, both warp splits, forward and backward."""
    test_psi_layer_edge_sizes(M, Q, Dout, N, True)
    test_psi_layer_edge_sizes(M, Q, Dout, N, False)


@pytest.mark.parametrize('N,M,Q', [(3, 1, 1), (5, 2, 3), (9, 67, 3), (200, 100, 4), (160, 128, 8), (5, 155, 2)])
def test_psi_derivatives_of_points_own_weights(N, M, Q):
    """Upstream weights of each point's own, not symmetric, at the sizes where their staging and
    the split change.  Same tolerance as the golden derivatives."""
    from geepee_gb300 import kernels as K
    rng = np.random.RandomState(N + M)
    Z, mu, S = rng.randn(M, Q), rng.randn(N, Q), rng.uniform(0.01, 1.0, (N, Q))
    lls2, lsf2 = rng.uniform(-0.5, 0.5, Q), np.array([0.3])
    d1, d2 = rng.randn(N, M), rng.randn(N, M, M) / M
    p1, p2 = O.psi_stats(lls2, lsf2, mu, S, Z)
    ell, sf2 = np.exp(0.5 * lls2), float(np.exp(lsf2[0]))
    got = K.compute_psi_derivatives(d1, p1, d2, p2, ell, sf2, mu, S, Z)
    ref = O.psi_derivatives(d1, p1, d2, p2, ell, sf2, mu, S, Z)
    for name, g, r in zip(('dsf2', 'dl', 'dZ', 'dmu', 'dS'), got, ref):
        assert_close(g, r, 1e-9, name)


@pytest.mark.parametrize('N', [1, 153, 330, 480, 777])
def test_psi_moments_where_the_tables_do_not_fit(N):
    """M = 200, one to six points a CTA (every number of points a pass): against the oracle, and a
    point's moments the same bits whatever the batch."""
    from geepee_gb300 import gpk
    M, Q = 200, 2
    rng = np.random.RandomState(5)
    Z, mu, S = rng.randn(M, Q), rng.randn(777, Q), rng.uniform(0.01, 1.0, (777, Q))
    A, B = rng.randn(1, M) / M, rng.randn(1, M, M) / M
    B = B + B.transpose(0, 2, 1)
    mu[2] = 40.0   # outside the fixed-point range
    lls2, lsf2 = np.array([0.2, -0.3]), np.array([0.3])
    def run(n):
        m, v = z(n, 1), z(n, 1)
        gpk.psi_fwd(dev(mu[:n]), dev(S[:n]), dev(Z), dev(lls2), dev(lsf2), dev(A), dev(B), m_out=m, v_out=v)
        return m, v
    m, v = run(N)
    p1, p2 = O.psi_stats(lls2, lsf2, mu[:N], S[:N], Z)
    m_ref = p1 @ A.T
    assert_close(m.cpu().numpy(), m_ref, TOL, 'm')
    assert_close(v.cpu().numpy(), np.exp(0.3) + np.einsum('dab,nab->nd', B, p2) - m_ref ** 2, TOL, 'v')
    m7, v7 = run(777)
    assert torch.equal(m, m7[:N]) and torch.equal(v, v7[:N])


@pytest.mark.parametrize('M,Q', [(10, 1), (50, 2), (30, 3), (100, 4), (120, 1)])
def test_psi_rollout_far_from_the_pseudo_inputs(M, Q):
    """One step from states ever farther from every pseudo-input: the mean stays good to its own sum of
    |terms|.  Its exponents e (base 2) are double-float sums, off by e 2^-46 each, the sum of M
    double-float terms by M 2^-46: (e + M) 2^-44 of sum |psi1 A|, as long as psi1 has not left the
    float range (e < 126)."""
    from geepee_gb300 import gpk
    rng = np.random.RandomState(M + Q)
    L = np.longdouble
    Z = rng.uniform(-1, 1, (M, Q))
    lls2, lsf2 = rng.uniform(-0.4, 0.1, Q), np.array([0.2])
    A = rng.randn(Q, M)
    B = rng.randn(Q, M, M) / M
    B = 0.1 * (B + B.transpose(0, 2, 1))
    l2, seen = np.exp(lls2.astype(L)), 0
    for far in np.linspace(3, 13, 21):
        mu, S = np.zeros(Q), rng.uniform(0.01, 0.05, Q)
        mu[0] = far * np.exp(0.5 * lls2[0])
        s1 = l2 + S.astype(L)
        e = 0.5 * ((mu.astype(L) - Z) ** 2 / s1).sum(1)
        p1 = np.exp(L(lsf2[0]) + 0.5 * np.log(l2 / s1).sum() - e)
        e2 = float(e.max()) / np.log(2.0)
        if e2 > 120:
            break
        seen += 1
        gm, _ = gpk.psi_rollout(dev(mu), dev(S), dev(Z), dev(lls2), dev(lsf2), dev(A), dev(B), 1)
        err = np.abs(gm[0].cpu().numpy() - A.astype(L) @ p1) / (np.abs(A).astype(L) @ p1)
        assert (err <= (e2 + M) * 2.0 ** -44).all(), (far, e2, err)
    assert seen >= 10
