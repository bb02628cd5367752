"""Thread-per-link kernels (NC <= 4): the FP64 exponential through
Cayley-Hamilton against the oracle's Taylor sum (every order, momenta that are
and are not Hermitian), the untuned register budget, and overlapped launches.

Tolerance: U' differs from the oracle's by roundings of sums of NC terms of
entries of modulus at most one, 1e-12 relative as for the other FP64 kernels."""
import numpy as np
import pytest

import askja_b200 as ab
from conftest import rel
from oracle import Oracle, fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hermitian", [True, False])
@pytest.mark.parametrize("nc", [2, 3, 4])
def test_fp64_exponential_every_order(nc, hermitian):
    dims = [3, 2, 2]
    rng = np.random.default_rng(11 * nc)
    O = Oracle(nc, dims)
    nl = O.vol * O.dim
    u = fields.haar(nc, nl, rng).reshape(O.shape)
    pi = np.asarray(fields.momenta(nc, nl, 2.0 * nc, rng, O)).reshape(O.shape)
    if not hermitian:
        pi = pi + 0.2 * (rng.standard_normal(O.shape) + 1j * rng.standard_normal(O.shape))
    for level in range(9):
        with ab.Engine(nc, dims, beta=4.0, level=level) as e:
            e.set_links(u)
            e.set_momenta(pi, 0)
            e.updateE(0.1)
            Pi = O.updateE(u, pi, 0.1)
            e.updateUandcopyDown(0.3)
            assert rel(e.get_links(), O.updateU(u, Pi, 0.3, level)) < 1e-12, level
            e.set_links(u)
            e.set_momenta(pi, 0)
            e.leapfrog(1, 0.2)  # the fused kernel
            want = O.updateU(u, O.updateE(u, pi, 0.1), 0.2, level)
            assert rel(e.get_links(), want) < 1e-12, level


# lattices on either side of the rules of default_occupancy and force_ahead
@pytest.mark.parametrize("nc,dims,precision", [(2, [24, 32, 26], "fp32"), (2, [23, 32, 25], "fp32"),
                                               (3, [24, 32, 26], "fp32"), (2, [64, 32, 32], "fp64"),
                                               (2, [65, 32, 32], "fp64"), (3, [16, 32, 18], "fp64"), (3, [17, 32, 18], "fp64"), (4, [24, 32, 26], "fp32")])
def test_register_budgets_give_the_same_fields(nc, dims, precision):
    out = []
    for occ in (None, 0, 1, 2):
        with ab.Engine(nc, dims, beta=2.0 * nc, dt=0.02, level=6, precision=precision, seed=5) as e:
            if occ is not None:
                ab.set_tuning(e, {"path": 0, "occupancy": occ})
            e.hot_start(3)
            e.run_trajectories(1, 2)
            out.append(e.get_links())
    for x in out[1:]:
        np.testing.assert_array_equal(x, out[0])


@pytest.mark.parametrize("nc,dims,precision", [(2, [6], "fp64"), (3, [4, 3, 2, 2, 3], "fp64"), (3, [4, 4, 4, 4], "fp32"),
                                               (4, [5, 4], "fp64"), (6, [3, 4], "fp32"), (16, [3, 3], "fp64")])
def test_overlapped_launches_replayed_or_not(nc, dims, precision):
    """A trajectory's kernels overlap their neighbours' starts; the fields are
    the same launched one by one, waited for in between, or replayed."""
    fieldsets = []
    for mode in ("graph", "eager", "stepwise"):
        with ab.Engine(nc, dims, beta=2.0 * nc, dt=0.02, level=6, precision=precision, reunitarise=False, seed=5) as e:
            e.hot_start(3)
            if mode != "stepwise":
                for _ in range(3):
                    last, _ = e.run_trajectories(1, 7, use_graph=mode == "graph")
                fieldsets.append((e.get_links(), e.get_momenta(0), last["h_new"]))
            else:
                e.initializeE(5, 0)
                e.leapfrog(7, 0.02)
                one = e.get_links()
                e.loadconfiguration()
                e.initializeE(5, 0)
                e.leapfrog(7, 0.02)
                np.testing.assert_array_equal(e.get_links(), one)
    np.testing.assert_array_equal(fieldsets[0][0], fieldsets[1][0])
    np.testing.assert_array_equal(fieldsets[0][1], fieldsets[1][1])
    assert fieldsets[0][2] == fieldsets[1][2]
