"""MD steps whose launches overlap their neighbours' starts, against the same steps
as single calls that each wait for the GPU: a load that came before its
launch's wait would read the links of the step before."""
import numpy as np
import pytest

import askja_b200 as ab

pytestmark = pytest.mark.gpu

STEPS, EPS = 7, 0.02


# grids of less than one wave and of several
@pytest.mark.parametrize("nc,dims,precision", [
    (2, [6], "fp64"), (2, [20, 20, 20, 12], "fp64"), (3, [8, 8, 8, 8], "fp64"), (3, [16, 16, 16, 12], "fp64"),
    (3, [4, 4, 4, 4], "fp32"), (3, [20, 20, 20, 12], "fp32"), (4, [12, 12, 12, 5], "fp64"), (3, [12, 12, 12, 5], "fp32-lean"),
    (5, [13, 12, 11], "fp64"), (6, [3, 4], "fp32"), (8, [8, 8, 8, 8], "fp32"), (16, [6, 6, 6], "fp64"), (24, [4, 4, 5], "fp32")])
def test_overlapped_steps_equal_single_calls(nc, dims, precision):
    # An entry is a sum of nc terms of modulus at most one, rounded some 16 times a
    # step (staples, exponential, product, projection) in either sequence; the
    # momenta grow to a few times that.  A link read a step late is off by eps P.
    tol = STEPS * 16 * nc * (1.2e-16 if precision == "fp64" else 6.0e-8)
    with ab.Engine(nc, dims, beta=2.0 * nc, dt=EPS, level=8, precision=precision, seed=5) as e:
        e.hot_start(3)
        e.takeconfiguration()
        e.initializeE(5, 0)
        e.updateE(0.5 * EPS)
        before = None
        for k in range(STEPS):
            before = e.get_links()
            e.updateUandcopyDown(EPS)
            e.updateE(EPS if k < STEPS - 1 else 0.5 * EPS)
        links, momenta = e.get_links(), e.get_momenta(1)
        assert np.abs(links - before).max() > 20 * tol
        for _ in range(3):
            e.loadconfiguration()
            e.initializeE(5, 0)
            e.leapfrog(STEPS, EPS)
            assert np.abs(e.get_links() - links).max() < tol
            assert np.abs(e.get_momenta(0) - momenta).max() < 4 * tol
