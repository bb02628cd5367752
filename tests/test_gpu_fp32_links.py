"""FP32 storage, NC >= 5 (warp MMA): every fused update projects the new links,
at any order of the exponential, and a force is no further from 64 bits than
FP32 FMAs put it."""
import time

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


@pytest.mark.parametrize("level", [1, 8])
def test_su32_drift_is_projected_and_cheap(level):
    """updateUandcopyDown of FP32 SU(32): one Newton-Schulz step in the update's own
    launch, no Gram-Schmidt pass, which took several times a whole fused step."""
    nc, dims, eps = 32, [4, 4, 4, 4], 0.02
    rng = np.random.default_rng(32)
    O = Oracle(nc, dims)
    nl = O.vol * O.dim
    u = fields.haar(nc, nl, rng).reshape(O.shape)
    pi = np.asarray(fields.momenta(nc, nl, 2.0 * nc, rng, O)).reshape(O.shape)
    with ab.Engine(nc, dims, beta=2.0 * nc, dt=eps, level=level, precision="fp32") as e:
        e.set_links(u)
        e.set_momenta(pi, 1)
        e.updateUandcopyDown(eps)
        assert rel(e.get_links(), projected_update(O, u, pi, eps, level)) < 1e-5
        np.testing.assert_array_equal(e.get_momenta(0), e.get_momenta(1))

        def median(f):
            t = []
            for _ in range(21):
                start = time.perf_counter()
                f()
                t.append(time.perf_counter() - start)
            return sorted(t)[10]

        # one fused update and one kick, against one update alone
        assert median(lambda: e.updateUandcopyDown(eps)) < median(lambda: e.leapfrog(1, eps))


def fma_force(u, dims):
    """-updateE(0 momenta, 1): the force of every link by FP32 FMAs in the order
    staple = (A B) C summed over planes, W = U S, emulated in 64 bits."""
    f32 = lambda x: x.astype(np.float32).astype(np.float64)

    def mac(c, a, b):
        re, im = c.real.copy(), c.imag.copy()
        for k in range(a.shape[-1]):
            x, y = a[..., :, k:k + 1], b[..., k:k + 1, :]
            re = f32(re + x.real * y.real)
            re = f32(re - x.imag * y.imag)
            im = f32(im + x.real * y.imag)
            im = f32(im + x.imag * y.real)
        return re + 1j * im

    exact = lambda c, a, b: c + a @ b
    d, nc = len(dims), u.shape[-1]
    links = [u[:, k].reshape(*dims, nc, nc) for k in range(d)]
    at = lambda x, step, axis: np.roll(x, -step, axis)
    out = []
    for prod in (exact, mac):
        f = np.zeros(u.shape, complex)
        for mu in range(d):
            s = np.zeros_like(links[0])
            for nu in range(d):
                if nu == mu:
                    continue
                far = at(links[nu], 1, mu)
                zero = np.zeros_like(s)
                s = prod(s, prod(zero, far, dagger(at(links[mu], 1, nu))), dagger(links[nu]))
                s = prod(s, prod(zero, dagger(at(far, -1, nu)), dagger(at(links[mu], -1, nu))), at(links[nu], -1, nu))
            w = prod(np.zeros_like(s), links[mu], s)
            w = w - dagger(w)
            w = w - np.trace(w, axis1=-2, axis2=-1)[..., None, None] / nc * np.eye(nc)
            f[:, mu] = (-0.5j * w).reshape(-1, nc, nc)
        out.append(f)
    return out


@pytest.mark.parametrize("dims", [[6, 8], [4, 3, 4], [3, 2, 3, 2]], ids=["2d", "3d", "4d"])
@pytest.mark.parametrize("nc", [5, 6, 7, 8, 9, 10, 11, 12, 15, 16, 17, 23, 24, 31, 40, 57])
def test_force_as_exact_as_fp32_fma(nc, dims):
    """Relative rms error of the force, no larger than that of FP32 FMAs; 5 % for
    the scatter of the rms of about 10^4 rounding errors (1 %) and for sums taken in
    another order."""
    rng = np.random.default_rng(700 + nc)
    O = Oracle(nc, dims)
    u = fields.haar(nc, O.vol * O.dim, rng).reshape(O.shape).astype(np.complex64).astype(np.complex128)
    zero = np.zeros_like(u)
    exact, fma = fma_force(u, dims)
    rms = lambda x: np.sqrt((np.abs(x) ** 2).mean())
    assert rms(O.updateE(u, zero, 1.0) + exact) < 1e-12 * rms(exact)
    with ab.Engine(nc, dims, beta=2.0 * nc, precision="fp32") as e:
        e.set_links(u)
        e.set_momenta(zero, 0)
        e.updateE(1.0)
        got = e.get_momenta(1)
    assert rms(got + exact) < 1.05 * rms(fma - exact)
