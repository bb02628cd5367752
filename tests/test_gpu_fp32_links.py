"""FP32 storage, NC >= 5 (warp MMA): every fused update projects the new links,
at any order of the exponential."""
import numpy as np
import pytest

import askja_b200 as ab
from conftest import rel
from oracle import Oracle, fields

pytestmark = pytest.mark.gpu


def dagger(x):
    return np.conj(np.swapaxes(x, -1, -2))


def projected_update(O, u, p, eps, level):
    """exp(i eps p) u, then the Newton-Schulz step v - (v v^dag - 1) v / 2."""
    v = O.updateU(u, p, eps, level)
    return 1.5 * v - 0.5 * (v @ dagger(v) @ v)


CASES = [(5, [3, 2, 3], 1), (6, [2, 3, 2], 2), (7, [3, 3], 3), (8, [3, 2, 2], 1), (8, [5, 3], 2), (12, [2, 3, 2], 1),
         (16, [3, 2], 2), (17, [2, 3], 1), (24, [2, 2], 3), (33, [2, 2], 1), (48, [2, 2], 2), (57, [2, 2], 1)]


@pytest.mark.parametrize("nc,dims,level", CASES, ids=[f"su{n}_{'x'.join(map(str, d))}_L{lv}" for n, d, lv in CASES])
def test_every_update_is_projected(nc, dims, level):
    """Three updates of step 0.1 with a Taylor sum far from unitary.  Tolerances of
    the other FP32 kernels' tests over as many updates: 1e-5 (links), 5e-5 (momenta)."""
    rng = np.random.default_rng(500 + nc)
    O = Oracle(nc, dims)
    nl = O.vol * O.dim
    u = fields.haar(nc, nl, rng).reshape(O.shape)
    pi = np.asarray(fields.momenta(nc, nl, 2.0 * nc, rng, O)).reshape(O.shape)
    eps = 0.1
    with ab.Engine(nc, dims, beta=2.0 * nc, dt=eps, level=level, precision="fp32") as e:
        e.set_links(u)
        e.set_momenta(pi, 0)
        e.leapfrog(3, eps)
        v, p = u, O.updateE(u, pi, eps / 2)
        for k in range(3):
            v = projected_update(O, v, p, eps, level)
            p = O.updateE(v, p, eps if k < 2 else eps / 2)
        assert rel(e.get_links(), v) < 1e-5
        assert rel(e.get_momenta(0), p) < 5e-5


@pytest.mark.parametrize("nc,dims", [(5, [3, 2, 2]), (8, [2, 3, 2]), (12, [2, 3]), (24, [2, 2])])
def test_first_update_of_a_trajectory_is_projected(nc, dims):
    """It runs in the launch that also sums the energies."""
    rng = np.random.default_rng(600 + nc)
    O = Oracle(nc, dims)
    u = fields.haar(nc, O.vol * O.dim, rng).reshape(O.shape)
    eps, level = 0.03, 1
    with ab.Engine(nc, dims, beta=2.0 * nc, dt=eps, level=level, precision="fp32", seed=11) as e:
        for traj in range(8):
            e.initializeE(11, traj)
            pi = e.get_momenta(0)
            e.set_links(u)
            if e.trajectory(1)["accepted"]:
                break
        else:
            pytest.fail("no trajectory was accepted")
        v = projected_update(O, u, O.updateE(u, pi, eps / 2), eps, level)
        assert rel(e.get_links(), v) < 1e-5
