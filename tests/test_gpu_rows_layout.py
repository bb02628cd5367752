"""Row-per-thread kernels (kernel_path 1) on link-major fields: the copies into the
tiles against the oracle at the sizes where they can go wrong (odd NC with its
padding column, a last CTA with few sites, every register bucket), and their cost."""
import time

import numpy as np
import pytest

import askja_b200 as ab
from conftest import rel
from oracle import Oracle, fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nc,dims", [(2, [5, 7]), (3, [3, 11]), (4, [33]), (5, [7, 3]), (6, [11, 2]), (7, [5, 5]), (8, [17, 2]),
                                     (9, [3, 3]), (13, [3, 3]), (16, [5, 2]), (17, [3, 2]), (31, [3]), (32, [2, 2]),
                                     (33, [2, 2]), (64, [2, 2])])
def test_copies_vs_oracle(nc, dims, precision):
    """FP64: sums of NC products of entries of unitary matrices, 1e-12 as for the other
    FP64 kernels; FP32: 1e-5 (links) and 5e-5 (momenta) after three updates."""
    rng = np.random.default_rng(900 + nc)
    O = Oracle(nc, dims)
    nl = O.vol * O.dim
    u = fields.near_identity(nc, nl, 0.5 / np.sqrt(nc), rng).reshape(O.shape)
    pi = np.asarray(fields.momenta(nc, nl, 2.0 * nc, rng, O)).reshape(O.shape)
    eps = 0.02
    with ab.Engine(nc, dims, beta=2.0 * nc, dt=eps, level=6, precision=precision, kernel_path=1) as e:
        e.set_links(u)
        e.set_momenta(pi, 0)
        e.leapfrog(3, eps)
        v, p = u, O.updateE(u, pi, eps / 2)
        for k in range(3):
            v = O.updateU(v, p, eps, 6)
            p = O.updateE(v, p, eps if k < 2 else eps / 2)
        tol_u, tol_p = (1e-12, 1e-12) if precision == "fp64" else (1e-5, 5e-5)
        assert rel(e.get_links(), v) < tol_u
        assert rel(e.get_momenta(0), p) < tol_p


def test_copies_are_coalesced():
    """FP32 SU(8) 10^4: a fused step (13 products and the copies) against the link update
    alone (8 products and a Gram-Schmidt pass).  1.2 times with links read row by row
    in the threads' order, 2.1 with threads a whole matrix apart."""
    with ab.Engine(8, [10] * 4, beta=16.0, dt=0.01, level=8, precision="fp32", kernel_path=1) as e:
        e.hot_start(1)
        e.initializeE(1, 0)
        e.updateE(0.01)

        def best(f):
            t = []
            for _ in range(15):
                start = time.perf_counter()
                f()
                t.append(time.perf_counter() - start)
            return sorted(t)[3]

        step = (best(lambda: e.leapfrog(21, 0.01)) - best(lambda: e.leapfrog(1, 0.01))) / 20
        assert step < 1.6 * best(lambda: e.updateUandcopyDown(0.01))
