"""Entry points called from two threads at once, on sizes whose launches differ."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(small, large, n=1500):
    """small() and large() n times each in two threads and streams; their exceptions and last results."""
    errors, last, gate = [], [None, None], threading.Barrier(2)

    def work(i, f):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                gate.wait()
                for _ in range(n):
                    last[i] = f()
            torch.cuda.synchronize()
        except Exception as e:
            errors.append(e)
    ts = [threading.Thread(target=work, args=(i, f)) for i, f in enumerate((small, large))]
    [t.start() for t in ts]
    [t.join() for t in ts]
    return errors, last


@pytest.mark.parametrize('op', ['contract', 'kern', 'gram', 'psi'])
def test_two_threads_two_sizes(op):
    """A call that needs little shared memory beside one that needs much, in kernels both share: neither
    launch is refused, and the results are those of the calls alone."""
    from geepee_gb300 import gpk
    g = torch.Generator(device='cuda').manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64, device='cuda')

    def make(n, m, d):
        x, z, l2, s2, A, B = r(n, d), r(m, d), r(d) * 0.1 + 1.0, r(1) * 0.1, r(1, m), r(1, m, m)
        B = 0.5 * (B + B.transpose(1, 2))
        if op == 'kern':
            return lambda: gpk.kern(x, z, l2, s2)
        if op == 'contract':
            k = torch.exp(-r(n, m).square())
            v = torch.empty((n, 1), dtype=torch.float64, device='cuda')
            return lambda: (gpk.det_contract(k, s2, A, B, v_out=v), v)[1]
        if op == 'gram':
            u, w, C = r(n, m), r(n, 1), torch.zeros((1, m, m), dtype=torch.float64, device='cuda')
            work = torch.empty(gpk.work_elems(gpk.OP_GRAM, n, m, 1, 1), dtype=torch.float64, device='cuda')
            return lambda: (C.zero_(), gpk.gram(u, u, w, C, work=work), C)[2]
        S, v = torch.exp(-r(n, d).square()), torch.empty((n, 1), dtype=torch.float64, device='cuda')
        return lambda: (gpk.psi_fwd(x, S, z, l2, s2, A, B, v_out=v), v)[1]

    small, large = {'kern': ((64, 20, 2), (64, 20, 40)), 'contract': ((8, 100, 1), (5000, 100, 1)),
                    'gram': ((16, 100, 1), (20000, 100, 1)), 'psi': ((2000, 20, 2), (2000, 50, 2))}[op]
    small, large = make(*small), make(*large)
    want = [small().clone(), large().clone()]
    torch.cuda.synchronize()
    errors, last = _both(small, large)
    assert not errors, errors
    assert torch.equal(last[0], want[0]) and torch.equal(last[1], want[1])
