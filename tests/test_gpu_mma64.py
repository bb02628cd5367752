"""FP64-MMA kernels (5 <= NC <= 64: link update, plaquette and kinetic sums on
link-major fields) against the FP64 oracle, at the edges of their 8 x 8 tiles:
one element beyond a tile, one short of it, whole tiles, every tile count, odd
colour numbers (no paired loads), one dimension (no staple), extent 1, link
counts that are no multiple of a CTA's.

Tolerances.  FP64: a result is at most a few dozen sums of NC products of
entries of unitary matrices, so 64 * NC * 2^-53 = 4.5e-13 at NC = 64; 1e-12
relative as for the other FP64 kernels.  FP32 storage: one rounding of 6e-8 per
stored entry and update; five updates and kicks of step 0.02 stay below 1e-5
(links) and 5e-5 (momenta), the bounds of the other FP32 kernels."""
import numpy as np
import pytest

import askja_b200 as ab
from conftest import rel
from oracle import Oracle, fields

pytestmark = pytest.mark.gpu

CASES = [(5, [3, 2, 3], 8), (5, [7], 6), (6, [2, 3, 1, 2], 6), (7, [3, 5], 3), (8, [3, 2, 2, 2], 8), (8, [5, 3], 0),
         (9, [2, 3], 8), (12, [2, 2, 3], 5), (15, [3, 2], 7), (16, [2, 1, 3, 2], 8), (17, [2, 3], 4), (24, [2, 3], 8),
         (31, [2, 2], 6), (32, [2, 3], 8), (33, [2, 2], 2), (40, [3, 2], 8), (48, [2, 2], 1), (57, [2, 2], 8),
         (64, [2, 3], 8)]
IDS = [f"su{n}_{'x'.join(map(str, d))}_L{lv}" for n, d, lv in CASES]


def start(nc, dims, seed):
    rng = np.random.default_rng(seed)
    O = Oracle(nc, dims)
    nl = O.vol * O.dim
    u = fields.near_identity(nc, nl, 0.5 / np.sqrt(nc), rng).reshape(O.shape)
    pi = fields.momenta(nc, nl, 2.0 * nc, rng, O)
    return O, u, np.asarray(pi).reshape(O.shape), rng


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nc,dims,level", CASES, ids=IDS)
def test_updates_and_sums_vs_oracle(nc, dims, level, precision):
    O, u, pi, _ = start(nc, dims, 100 + nc)
    tol_u, tol_p, tol_h = (1e-12, 1e-12, 1e-12) if precision == "fp64" else (1e-5, 5e-5, 1e-5)
    eps = 0.02
    with ab.Engine(nc, dims, beta=2.0 * nc, dt=eps, level=level, precision=precision, reunitarise=False) as e:
        if precision == "fp32" and nc in (32, 64):
            ab.set_tuning(e, {"path": 4})  # the default there is the TF32 tensor-core path
        e.set_links(u)
        e.set_momenta(pi, 0)
        assert e.EnergyMag() == pytest.approx(O.EnergyMag(u), rel=tol_h, abs=tol_h * O.vol)
        assert e.simpleenergyEl(0) == pytest.approx(O.simpleenergyEl(pi), rel=tol_h)
        e.leapfrog(3, eps)
        uu, pp = u, O.updateE(u, pi, eps / 2)
        for k in range(3):
            uu = O.updateU(uu, pp, eps, level)
            pp = O.updateE(uu, pp, eps if k < 2 else eps / 2)
        assert rel(e.get_links(), uu) < tol_u
        assert rel(e.get_momenta(0), pp) < tol_p
        # out of place, then the separate link update
        e.updateE(eps)
        e.updateUandcopyDown(eps)
        pp = O.updateE(uu, pp, eps)
        uu = O.updateU(uu, pp, eps, level)
        assert rel(e.get_momenta(1), pp) < tol_p
        assert rel(e.get_momenta(0), pp) < tol_p
        assert rel(e.get_links(), uu) < tol_u


@pytest.mark.parametrize("nc", [5, 8, 17, 33])
def test_momenta_need_not_be_hermitian(nc):
    """The link update takes any matrix for P, as the reference's mexpi does."""
    O, u, pi, rng = start(nc, [2, 2], 7 + nc)
    pi = pi + 0.3 * (rng.standard_normal(pi.shape) + 1j * rng.standard_normal(pi.shape))
    for level in (2, 6, 8):
        with ab.Engine(nc, [2, 2], beta=5.0, level=level) as e:
            e.set_links(u)
            e.set_momenta(pi, 1)
            e.updateUandcopyDown(0.05)
            assert rel(e.get_links(), O.updateU(u, pi, 0.05, level)) < 1e-12
            assert e.simpleenergyEl(1) == pytest.approx(O.simpleenergyEl(pi), rel=1e-12)


@pytest.mark.parametrize("nc", [6, 16, 33])
def test_reunitarise_after_each_update_fp64(nc):
    """reunitarise = 1 in FP64: the full projection after every link update."""
    O, u, pi, _ = start(nc, [3, 2], 50 + nc)
    with ab.Engine(nc, [3, 2], beta=5.0, level=4, reunitarise=True) as e:
        e.set_links(u)
        e.set_momenta(pi, 1)
        e.updateUandcopyDown(0.3)  # far from unitary at this order
        want = O.reunitarise(O.updateU(u, pi, 0.3, 4).reshape(-1, nc, nc)).reshape(O.shape)
        assert rel(e.get_links(), want) < 1e-11


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nc,dims", [(33, [5, 15]), (40, [7, 11]), (45, [75, 1]), (48, [5, 5, 2])])
def test_more_links_than_processors(nc, dims, precision):
    """33 <= NC <= 48 above 148 links: two CTAs per SM under the tight register budget."""
    O, u, pi, _ = start(nc, dims, 300 + nc)
    tol_u, tol_p = (1e-12, 1e-12) if precision == "fp64" else (1e-5, 5e-5)
    with ab.Engine(nc, dims, beta=2.0 * nc, dt=0.02, level=8, precision=precision, reunitarise=False) as e:
        e.set_links(u)
        e.set_momenta(pi, 0)
        e.leapfrog(1, 0.02)
        p = O.updateE(u, pi, 0.01)
        v = O.updateU(u, p, 0.02, 8)
        assert rel(e.get_links(), v) < tol_u
        assert rel(e.get_momenta(0), O.updateE(v, p, 0.01)) < tol_p


@pytest.mark.parametrize("nc", [5, 8, 11, 16, 23, 31, 40, 57, 63])
def test_split_products_keep_32_bits(nc):
    """FP32 storage multiplies in TF32 split in two; one part alone is off by 2^-12.

    With u = 2^-24, a split product drops less than u, rounds once per 8 columns
    and once per stored operand: (NT + 3) u a product.  A kick of far-from-unit
    links is three products and four rounded links, its anti-hermitian part
    1 / sqrt(2) of the whole: 1.5 (3 (NT + 3) + 4) u.  An update with |X| of order
    one rounds U on the way in and out, its increment (LEVEL products, falling as
    1 / k!) to 2 (NT + 3) u: (2 (NT + 3) + 4) u."""
    dims = [3, 2, 2]
    O, u, _, rng = start(nc, dims, 70 + nc)
    u = fields.near_identity(nc, u.size // nc ** 2, 2.0 / np.sqrt(nc), rng).reshape(O.shape)
    pi = np.asarray(fields.momenta(nc, u.size // nc ** 2, 2.0 * nc, rng, O)).reshape(O.shape)
    nt, unit = (nc + 7) // 8, 2.0 ** -24
    with ab.Engine(nc, dims, beta=2.0 * nc, dt=0.1, level=8, precision="fp32", reunitarise=False) as e:
        ab.set_tuning(e, {"path": 4})
        e.set_links(u)
        e.set_momenta(np.zeros_like(pi), 0)
        e.updateE(0.1)
        assert rel(e.get_momenta(1), O.updateE(u, np.zeros_like(pi), 0.1)) < 1.5 * (3 * (nt + 3) + 4) * unit
        e.set_momenta(0.5 * pi, 1)
        e.updateUandcopyDown(0.1)
        assert rel(e.get_links(), O.updateU(u, 0.5 * pi, 0.1, 8)) < (2 * (nt + 3) + 4) * unit


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_batch_equals_single_chains(precision):
    chains = [dict(nc=nc, dims=d, beta=2.0 * nc, dt=0.02, level=lv, seed=40 + nc)
              for nc, d, lv in [(5, [3, 5, 3], 8), (8, [3, 3, 3], 6), (12, [2, 3, 2], 8), (16, [3, 3], 8),
                                (8, [5, 2], 7), (33, [2, 2], 6)]]
    chains.append(dict(nc=3, dims=[4, 4], beta=5.0, dt=0.02, level=6, seed=3))
    with ab.Batch(chains, precision=precision) as b:
        b.hot_start(9)
        starts = [b.get_links(c) for c in range(len(chains))]
        res = b.run(2, 3)
        ends = [b.get_links(c) for c in range(len(chains))]
    for c, ch in enumerate(chains):
        with ab.Engine(ch["nc"], ch["dims"], beta=ch["beta"], dt=ch["dt"], level=ch["level"], precision=precision,
                       seed=ch["seed"]) as e:
            e.set_links(starts[c])
            last, _ = e.run_trajectories(2, 3)
            for k in ("h_old", "h_new", "u", "accepted", "n_acc"):
                assert res[c][k] == last[k], (c, k)
            np.testing.assert_array_equal(ends[c], e.get_links())


@pytest.mark.parametrize("nc,dims", [(2, [40, 3]), (3, [33, 2, 2]), (3, [65]), (4, [1, 5, 4]), (4, [97, 2]), (5, [4, 3]),
                                     (8, [3, 2, 3]), (13, [2, 4]), (24, [2, 3]), (33, [3, 2]), (64, [2, 2])])
def test_lines_gauss_and_unitarity_vs_oracle(nc, dims):
    """Line products shared between lanes (NC <= 4: extents around 32 and 64
    links) or walked by the MMA, the Gauss law's grouped sums, UViol of links
    that are not unitary, and the one-read-back measure()."""
    O, u, pi, rng = start(nc, dims, 3 * nc)
    u = u * (1.0 + 0.01 * rng.standard_normal(u.shape))
    with ab.Engine(nc, dims, beta=2.0 * nc, precision="fp64") as e:
        e.set_links(u)
        e.set_momenta(pi, 0)
        e.updateE(0.05)
        Pi = O.updateE(u, pi, 0.05)
        one = {"WilsonLoop": (e.WilsonLoop(), O.WilsonLoop_sun(u)), "GaussLaw": (e.GaussLaw(), O.GaussLaw(u, Pi)),
               "UViol": (e.UViol(), O.UViol(u)), "EnergyEl": (e.EnergyEl(), O.EnergyEl(pi, Pi))}
        if len(dims) > 1:
            one["Polyakov"] = (e.PolyakovLoop(), O.PolyakovLoop(u))
            one["slices"] = (e.scalarLoopcorr(), O.scalarLoopcorr(u))
            for d in range(1, len(dims)):
                one[f"Wilson{d}"] = (e.WilsonLoopDir(d), O.WilsonLoopDir(u, d))
            t, s = e.PlaqExp()
            want = [t, s, e.PolyakovLoop()] + [e.WilsonLoopDir(d) for d in range(1, len(dims))]
            want += [e.GaussLaw(), e.UViol()]
            np.testing.assert_array_equal(e.measure(), want)
        for name, (got, ref) in one.items():
            # a line of n links multiplies the rounding of n products; the links' norms stray by 1 %
            np.testing.assert_allclose(got, ref, rtol=1e-11, atol=1e-12, err_msg=name)


@pytest.mark.parametrize("nc", [6, 16, 40])
def test_counted_ranges_add_up(nc):
    O, u, pi, _ = start(nc, [5, 3], nc)
    with ab.Engine(nc, [5, 3], beta=3.0) as e:
        e.set_links(u)
        e.set_momenta(pi, 0)
        whole = np.array([e.EnergyMag(), e.simpleenergyEl(0)])
        parts = np.zeros(2)
        for s0, s1 in ((0, 4), (4, 5), (5, 15)):
            e.set_reduction_range(s0, s1)
            parts += [e.EnergyMag(), e.simpleenergyEl(0)]
        np.testing.assert_allclose(parts, whole, rtol=1e-12)
