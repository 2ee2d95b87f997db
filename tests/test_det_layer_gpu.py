"""The deterministic-input layer at the edges of its fixed-point and digit forms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device='cuda').contiguous()


@pytest.mark.parametrize('n,m,d,dout', [(1, 1, 1, 1), (17, 15, 2, 2), (33, 16, 16, 1), (70, 129, 3, 4), (50, 200, 8, 2),
                                        (31, 255, 5, 1), (5000, 103, 8, 2)])
def test_det_layer_fixed_point_edges(n, m, d, dout):
    """The fixed-point kernel rows and the digit contraction at the edges of their tiles, with rows
    whose coordinates leave the fixed-point range, rows that are zero or NaN, columns of B from
    1e-25 to 1e25 and a zero column.  The rows: 2^-45 (|a| + 1) of an entry with exponent a (the
    double-float form's error, the larger one).  The contraction, from the device's own rows: each product is off by at most
    2^-47 of the row's largest times the column's largest."""
    from geepee_gb300 import gpk
    rng = np.random.RandomState(n + m)
    L = np.longdouble
    x, z = rng.randn(n, d), rng.randn(m, d)
    if n > 16:
        x[3] = z[5 % m] + 60.0      # far from every z: coordinates out of range, rows zero
        x[7] = np.nan
        x[11] = 1e12
        x[13] = z[m - 1] + 1e-9
    if m > 16:
        z[9] = 25.0                 # a column out of range
        if n > 16:
            x[14] = z[9] + 0.1
    l2, s2 = np.log(rng.uniform(0.5, 2.0, d) * d), np.array([0.3])
    A, B = rng.randn(dout, m), rng.randn(dout, m, m) * 10.0 ** rng.uniform(-25, 25, (dout, 1, m))
    B[:, :, m // 2] = 0.0
    e = lambda *s: torch.full(s, -7.0, dtype=torch.float64, device='cuda')
    kfu, Bk, mo, vo = e(n, m), e(n, dout, m), e(n, dout), e(n, dout)
    At, Bt, s2t = dev(A), dev(B), dev(s2)
    gpk.det_fwd(dev(x), dev(z), dev(l2), s2t, At, Bt, kfu, Bk, mo, vo)
    K = gpk.kern(dev(x), dev(z), dev(l2), s2t)
    assert torch.equal(torch.nan_to_num(K, nan=-1.0), torch.nan_to_num(kfu, nan=-1.0))
    nan = np.isnan(x).any(1)
    a = (s2[0] - 0.5 * ((x[:, None].astype(L) - z[None]) ** 2 / np.exp(l2.astype(L))).sum(-1))[~nan]
    k, Kg = np.exp(a), K.cpu().numpy()
    assert np.isnan(Kg[nan]).all()
    err = np.abs(Kg[~nan] - k)
    assert (err <= 2.0 ** -45 * (np.abs(a) + 1) * k + 1e-37).all(), float((err / (k + 1e-300)).max())
    kg = Kg[~nan].astype(L)
    bk = np.einsum('na,dab->ndb', kg, B.astype(L))
    km, bm = kg.max(1), np.abs(B).max(1)
    g = Bk.cpu().numpy()
    assert np.isnan(g[nan]).all() and np.isnan(mo.cpu().numpy()[nan]).all() and np.isnan(vo.cpu().numpy()[nan]).all()
    assert (np.abs(g[~nan] - bk) <= m * 2.0 ** -47 * km[:, None, None] * bm[None] + 1e-37).all()
    mm = np.einsum('na,da->nd', kg, A.astype(L))
    assert (np.abs(mo.cpu().numpy()[~nan] - mm) <= m * 2.0 ** -47 * km[:, None] * np.abs(A).max(1)[None] + 1e-37).all()
    vv = np.exp(L(s2[0])) + np.einsum('nb,ndb->nd', kg, bk)
    vs = 2 + m * m * (km[:, None] ** 2 * bm.max(1)[None])
    assert (np.abs(vo.cpu().numpy()[~nan] - vv) <= 2.0 ** -46 * vs).all()
    if gpk.det_contract_supported(torch.float64, m, dout):
        hi = B.astype(np.float32)
        pairs = dev(np.stack([hi, (B - hi).astype(np.float32)], -1).astype(np.float32).view(np.float64)[..., 0])
        got = []
        for Bp, flag in ((Bt, False), (pairs, True)):
            Bk2, m2, v2 = e(n, dout, m), e(n, dout), e(n, dout)
            gpk.det_contract(kfu, s2t, At, Bp, Bk2, m2, v2, b_pairs=flag)
            got.append([torch.nan_to_num(t, nan=-1.0) for t in (Bk2, m2, v2)])
            assert (np.abs(Bk2.cpu().numpy()[~nan] - bk) <= m * 2.0 ** -47 * km[:, None, None] * bm[None] + 1e-37).all()
        assert all(torch.equal(p, q) for p, q in zip(*got))
        assert torch.equal(got[0][1], torch.nan_to_num(mo, nan=-1.0))


@pytest.mark.parametrize('n,m,dout', [(1, 1, 1), (15, 7, 2), (16, 8, 1), (17, 16, 4), (129, 33, 3), (1000, 104, 1),
                                      (3001, 100, 2), (700, 129, 2), (97, 255, 1), (40, 460, 1)])
def test_symmetric_gram_edges(n, m, dout):
    """The digit form of the symmetric weighted Gram reduction at the edges of its tiles and row
    chunks (the last size takes the pair form), columns from 1e-15 to 1e15, weights over twelve
    decades with zeros, and a column with an infinity.  Every product is off by at most 2^-47 of
    the largest |w u_a| times the largest |u_b|."""
    from geepee_gb300 import gpk
    rng = np.random.RandomState(n + m)
    L = np.longdouble
    u = rng.randn(n, m) * 10.0 ** rng.uniform(-15, 15, m)
    w = rng.randn(n, dout) * 10.0 ** rng.uniform(-6, 6, (n, dout))
    w[n // 2] = 0.0
    if m > 8:
        u[:, 5] = 0.0
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device='cuda')
    work = z(gpk.work_elems(gpk.OP_GRAM, n, m, 1, dout))
    ref = np.einsum('nd,na,nb->dab', w.astype(L), u.astype(L), u.astype(L))
    ua = np.abs(u).max(0)
    wa = np.abs(w[:, :, None] * u[:, None]).max(0)
    tol = n * 2.0 ** -47 * np.maximum(wa[:, :, None] * ua, wa[:, None] * ua[:, None]) + 1e-37
    C = z(dout, m, m)
    ut = dev(u)
    gpk.gram(ut, ut, dev(w), C, work=work)
    assert (np.abs(C.cpu().numpy() - ref) <= tol).all()
    if m > 8:
        u[n // 3, 6] = np.inf
        C, ut = z(dout, m, m), dev(u)
        gpk.gram(ut, ut, dev(w), C, work=work)
        g, keep = C.cpu().numpy(), np.arange(m) != 6
        assert not np.isfinite(g[:, 6]).any() and not np.isfinite(g[:, :, 6]).any()
        assert (np.abs(g - ref) <= tol)[:, keep][:, :, keep].all()


def test_gram_workspace_of_a_larger_call():
    """A workspace sized for the largest call serves every smaller one (fewer rows are split into more
    chunks than twenty thousand are)."""
    from geepee_gb300 import gpk
    rng = np.random.RandomState(2)
    m = 20
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device='cuda')
    for dout in (1, 3):
        work = z(gpk.work_elems(gpk.OP_GRAM, 20000, m, 1, 3))
        for n in (1, 16, 800, 2432, 2433, 4865):
            u, w = rng.randn(n, m), rng.randn(n, dout)
            C, ut = z(dout, m, m), dev(u)
            gpk.gram(ut, ut, dev(w), C, work=work)
            ref = np.einsum('nd,na,nb->dab', w, u, u)
            assert np.abs(C.cpu().numpy() - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize('bits', [-1, 0x7fffffffffffffff, 0x7ff8000000000000, 0x7ff0000000000001])
def test_contraction_of_any_nan(bits):
    """A NaN of any payload (all ones among them) in B or A makes its column of Bk or its output's m NaN,
    and v through B; the rest stays finite."""
    from geepee_gb300 import gpk
    rng = np.random.RandomState(4)
    n, m = 20, 30
    k, A, B = np.exp(-rng.rand(n, m)), rng.randn(2, m), rng.randn(2, m, m)
    nan = np.array([bits], dtype=np.int64).view(np.float64)
    B[0, 3, 7], A[1, 5] = nan[0], nan[0]
    e = lambda *s: torch.zeros(s, dtype=torch.float64, device='cuda')
    Bk, mo, vo = e(n, 2, m), e(n, 2), e(n, 2)
    gpk.det_contract(dev(k), dev([0.1]), dev(A), dev(B), Bk, mo, vo)
    want = np.zeros((2, m), bool)
    want[0, 7] = True
    assert (np.isnan(Bk.cpu().numpy()) == want).all()
    assert (np.isnan(mo.cpu().numpy()) == [False, True]).all()
    assert (np.isnan(vo.cpu().numpy()) == [True, False]).all()


def _graded(kind, n, m, rng):
    """Kernel rows over six lengthscales and a B whose size grows against them."""
    z, x = np.sort(rng.uniform(0, 6, m)), rng.uniform(0, 1.5, n)
    k = np.exp(-0.5 * (x[:, None] - z) ** 2)
    C = rng.uniform(0.5, 1, (m, m)) * rng.choice([-1.0, 1.0], (m, m))
    g = 10.0 ** (2 * z)                       # 1 to 1e12, along the decay of k
    if kind == 'rows':
        return k, g[:, None] * C
    C = 0.5 * (C + C.T)
    if kind == 'columns':
        return k, C * g
    if kind == 'symmetric':
        return k, g[:, None] * C * g
    if kind == 'diagonal':                    # far pseudo-inputs coupled to themselves alone
        return k, np.diag(np.where(z > 3, 1e20, 1.0))
    if kind == 'local':                       # most kernel values below the float range
        return np.exp(-0.5 * (x[:, None] - z) ** 2 * 60), np.diag(rng.uniform(1, 4, m)) + 0.1 * C
    return k, np.where(C == np.diag(np.diag(C)), 0.0, C * 1e-3) + np.diag(g)   # 'mixed'


@pytest.mark.parametrize('m', [7, 60, 130, 201])
@pytest.mark.parametrize('kind', ['rows', 'columns', 'symmetric', 'diagonal', 'local', 'mixed'])
def test_contraction_of_graded_weights(kind, m):
    """Weights graded against the kernel rows keep the double-float form's accuracy: m and v to
    their sums of |terms| (a sum of M double-float terms: M 2^-47 of it; v's digit products, trusted
    where the weighted sums of |k B| reach a sixteenth of the scales, another 16 M 2^-50.6), Bk to
    M 2^-50 of the scales' product beside its own M 2^-47, and where B is dense that is its sum of
    |terms| too."""
    from geepee_gb300 import gpk
    rng = np.random.RandomState(m)
    L = np.longdouble
    n = 40
    k, B = _graded(kind, n, m, rng)
    A = 10.0 ** (np.argsort(np.argsort(k[0])) * (-12.0 / m)) * rng.randn(1, m)
    e = lambda *s: torch.zeros(s, dtype=torch.float64, device='cuda')
    Bk, mo, vo = e(n, 1, m), e(n, 1), e(n, 1)
    if m <= 128:
        gpk.det_contract(dev(k), dev([0.0]), dev(A), dev(B[None]), Bk, mo, vo)
        kg = k
    else:   # through the fused entry point, whose rows are its own
        kd = e(n, m)
        x = rng.uniform(0, 1.5, (n, 1))
        z = np.sort(rng.uniform(0, 6, m))[:, None]
        l2 = np.zeros(1) if kind != 'local' else np.full(1, -np.log(60.0))
        gpk.det_fwd(dev(x), dev(z), dev(l2), dev([0.0]), dev(A), dev(B[None]), kd, Bk, mo, vo)
        kg = kd.cpu().numpy()
    kg, Bl = kg.astype(L), B.astype(L)
    S = np.abs(kg) @ np.abs(Bl)
    bk, tiny = kg @ Bl, 1e-36
    sm = (np.abs(kg) @ np.abs(A.astype(L)).T)[:, 0]
    assert (np.abs(mo.cpu().numpy()[:, 0] - (kg @ A.astype(L).T)[:, 0]) <= (m + 16) * 2.0 ** -47 * sm + tiny).all()
    T = (S * np.abs(kg)).sum(1)
    dv = np.abs(vo.cpu().numpy()[:, 0] - (1 + (bk * kg).sum(1)))
    assert (dv <= (3 * m + 16) * 2.0 ** -47 * (T + 1) + 16 * m * 2.0 ** -50.6 * T).all(), float((dv / (T + 1)).max())
    c = np.abs(Bl).max(0)
    r = (np.abs(Bl) / np.where(c > 0, c, 1)).max(1)
    scale = (kg * r).max(1)[:, None] * c
    db = np.abs(Bk.cpu().numpy()[:, 0] - bk)
    # (the scales are powers of two up to four times c r, twice each)
    assert (db <= m * 2.0 ** -48 * scale + (m + 16) * 2.0 ** -47 * S + tiny).all()
    if kind in ('rows', 'columns', 'symmetric'):
        assert (db <= 8 * m * 2.0 ** -48 * S).all(), float((db / S).max())


@pytest.mark.parametrize('n,m,dout', [(40, 12, 1), (129, 33, 2), (3000, 100, 1)])
@pytest.mark.parametrize('p', [-2, -1, 1, 4])
def test_gram_of_graded_rows(n, m, dout, p):
    """Rows that grow over twelve decades with weights that grow as a power of them: every sum is good to
    its sum of |terms| (n 2^-47 of it, as a sum of n double-float terms; the columns are dense)."""
    from geepee_gb300 import gpk
    rng = np.random.RandomState(n + m)
    L = np.longdouble
    g = 10.0 ** rng.uniform(-6, 6, (n, 1))
    u = g * rng.uniform(0.5, 1, (n, m)) * rng.choice([-1.0, 1.0], (n, m))
    w = g ** p * rng.uniform(0.5, 1, (n, dout)) * rng.choice([-1.0, 1.0], (n, dout))
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device='cuda')
    C, ut = z(dout, m, m), dev(u)
    gpk.gram(ut, ut, dev(w), C, work=z(gpk.work_elems(gpk.OP_GRAM, n, m, 1, dout)))
    ref = np.einsum('nd,na,nb->dab', w.astype(L), u.astype(L), u.astype(L))
    S = np.einsum('nd,na,nb->dab', np.abs(w).astype(L), np.abs(u).astype(L), np.abs(u).astype(L))
    err = np.abs(C.cpu().numpy() - ref)
    assert (err <= n * 2.0 ** -47 * S).all(), float((err / S).max())


@pytest.mark.parametrize('n,m,d', [(1, 1, 1), (50, 17, 2), (33, 129, 5), (300, 100, 8)])
@pytest.mark.parametrize('shift', [64.0, 2000.0, 1.7e9])
def test_kernel_rows_do_not_depend_on_the_origin(n, m, d, shift):
    """Kernel rows of inputs and pseudo-inputs translated together (by exact amounts: multiples of 2^-20) are the
    same to the fixed point's last places: each coordinate is off by at most 2^-55 either time, which is
    4 2^-55 sum |x - z| <= 4 2^-55 16 sqrt(d) in an exponent below 256, beside its own 2^-51 d; the exponential's
    error is below 2^-49."""
    from geepee_gb300 import gpk
    rng = np.random.RandomState(n + d)
    q = lambda a: np.round(a * 2.0 ** 20) / 2.0 ** 20
    x, z = q(4 * rng.randn(n, d)), q(4 * rng.randn(m, d))
    l2, s2 = dev(rng.uniform(-0.5, 0.5, d) + np.log(d)), dev([0.2])
    K = gpk.kern(dev(x), dev(z), l2, s2).cpu().numpy()
    off = shift * (1 - 2 * (np.arange(d) % 2))
    Ks = gpk.kern(dev(x + off), dev(z + off), l2, s2).cpu().numpy()
    tol = 2 * (2.0 ** -49 + 16 * d ** 0.5 * 2.0 ** -53 + d * 2.0 ** -51)
    assert (np.abs(Ks - K) <= tol * K + 1e-300).all(), float((np.abs(Ks - K) / np.maximum(K, 1e-300)).max())


@pytest.mark.parametrize('span', [40.0, 1000.0, 60000.0, 1e6])
def test_kernel_rows_over_a_wide_range(span):
    """A one-dimensional range of many lengthscales, with inputs far outside it: each entry to
    2^-45 (|a| + 1) of itself (a its exponent), zero where it is below the float range."""
    from geepee_gb300 import gpk
    rng = np.random.RandomState(3)
    L = np.longdouble
    z = np.sort(rng.uniform(0, span, 150))[:, None]
    x = np.concatenate([z[:, 0] + 3 * rng.randn(150), rng.uniform(0, span, 200), [-1e9, 1e12, 1e200, 7 * span]])[:, None]
    K = gpk.kern(dev(x), dev(z), dev([0.0]), dev([0.4])).cpu().numpy()
    a = 0.4 - 0.5 * (x.astype(L) - z.astype(L).T) ** 2
    k = np.exp(a)
    assert (np.abs(K - k) <= 2.0 ** -45 * (np.abs(a) + 1) * k + 1e-37).all()
    assert (K[-4:] == 0).all()
    Kn = gpk.kern(dev([[np.nan], [0.5]]), dev(z), dev([0.0]), dev([0.4])).cpu().numpy()
    assert np.isnan(Kn[0]).all() and np.isfinite(Kn[1]).all()


@pytest.mark.parametrize('n,m,dout', [(17, 9, 1), (130, 40, 2), (2000, 100, 1), (5000, 129, 2)])
@pytest.mark.parametrize('kind', ['local', 'mixed', 'disjoint'])
def test_gram_of_columns_that_hardly_meet(n, m, dout, kind):
    """Kernel rows of a layer whose lengthscale is short against the spread of its pseudo-inputs: the sums of
    far pseudo-inputs are tens of decades below the near ones' and each is still good to n 2^-47 of its own
    sum of |terms|."""
    from geepee_gb300 import gpk
    rng = np.random.RandomState(n + m)
    L = np.longdouble
    z, x = np.sort(rng.uniform(0, 1, m)), rng.uniform(0, 1, n)
    u = np.exp(-0.5 * (x[:, None] - z) ** 2 / 0.06 ** 2)
    if kind == 'mixed':                            # broad columns among the narrow ones
        u[:, ::3] = np.exp(-0.5 * (x[:, None] - z[::3]) ** 2)
    if kind == 'disjoint':                         # every other column on rows of its own, and a column of zeros
        u[::2, ::2] = 0.0
        u[1::2, 1::2] *= 1e-9
        u[:, m // 2] = 0.0
    w = rng.randn(n, dout)
    z0 = lambda *s: torch.zeros(s, dtype=torch.float64, device='cuda')
    C, ut = z0(dout, m, m), dev(u)
    gpk.gram(ut, ut, dev(w), C, work=z0(gpk.work_elems(gpk.OP_GRAM, n, m, 1, dout)))
    ref = np.einsum('nd,na,nb->dab', w.astype(L), u.astype(L), u.astype(L))
    S = np.einsum('nd,na,nb->dab', np.abs(w).astype(L), u.astype(L), u.astype(L))
    err = np.abs(C.cpu().numpy() - ref)
    assert (err <= n * 2.0 ** -47 * S + 1e-37).all(), float((err / (S + 1e-37)).max())
    u[n // 3, m // 2] = np.nan                     # a NaN in a column of zeros
    C, ut = z0(dout, m, m), dev(u)
    gpk.gram(ut, ut, dev(w), C, work=z0(gpk.work_elems(gpk.OP_GRAM, n, m, 1, dout)))
    g, keep = C.cpu().numpy(), np.arange(m) != m // 2
    assert np.isnan(g[:, m // 2]).all() and np.isnan(g[:, :, m // 2]).all() and np.isfinite(g[:, keep][:, :, keep]).all()


@pytest.mark.parametrize('kind', ['rows', 'diagonal', 'mixed'])
def test_contraction_of_graded_pairs(kind):
    """The same weights as double-float pairs give the same bits, the rows formed again in double-float
    among them."""
    from geepee_gb300 import gpk
    m, n = 60, 40
    rng = np.random.RandomState(m)
    k, B = _graded(kind, n, m, rng)
    A = rng.randn(1, m)
    hi = B.astype(np.float32)
    pairs = np.stack([hi, (B - hi).astype(np.float32)], -1).astype(np.float32).view(np.float64)[..., 0]
    got = []
    for Bp, flag in ((B, False), (pairs, True)):
        out = [torch.zeros(s, dtype=torch.float64, device='cuda') for s in ((n, 1, m), (n, 1), (n, 1))]
        gpk.det_contract(dev(k), dev([0.0]), dev(A), dev(Bp[None]), *out, b_pairs=flag)
        got.append(out)
    assert all(torch.equal(p, q) for p, q in zip(*got))


@pytest.mark.parametrize('m', [16, 33, 100, 255])
@pytest.mark.parametrize('above', [0, 1])
def test_gram_where_the_digits_begin(m, above):
    """The last size of the pair form and the first of the digit form: N M (M + 1) / 2 at and above 2^20."""
    from geepee_gb300 import gpk
    n = (1 << 20) // (m * (m + 1) // 2) + above
    rng = np.random.RandomState(m)
    L = np.longdouble
    u, w = np.exp(-rng.rand(n, m) * 8), rng.randn(n, 1)
    z0 = lambda *s: torch.zeros(s, dtype=torch.float64, device='cuda')
    C, ut = z0(1, m, m), dev(u)
    gpk.gram(ut, ut, dev(w), C, work=z0(gpk.work_elems(gpk.OP_GRAM, n, m, 1, 1)))
    ref = (u.astype(L) * w).T @ u.astype(L)
    S = (u.astype(L) * np.abs(w)).T @ u.astype(L)
    assert (np.abs(C.cpu().numpy()[0] - ref) <= n * 2.0 ** -47 * S).all()
