"""Reductions whose total is added up by the last block or, from a number of
blocks on, by a launch of its own, and the slice averages of link-major fields,
against plain torch in 64 bits on the engine's own fields.

Tolerance: sums of at most 2e7 terms in FP64, whatever the order, are within
2e7 * 1.1e-16 of their terms' absolute sum in the worst case, and the terms are
of one sign (tr P^2, squared moduli) or of order one (1 - ReTr P / N): 1e-8.
UViol is of the links' rounding, with products of N terms: relative to (N u)^2 per
link in FP64 its own rounding, so it is compared where links are scaled off
U(N)."""
import numpy as np
import pytest

import askja_b200 as ab

pytestmark = pytest.mark.gpu


def torch_sums(u, p, dims, nc):
    import torch

    u = torch.from_numpy(u).cuda().view(*dims, len(dims), nc, nc)
    p = torch.from_numpy(p).cuda().view(-1, nc, nc)
    d = len(dims)
    both = [0.0, 0.0]
    for mu in range(d):
        for nu in range(mu + 1, d):
            a = u[..., mu, :, :] @ torch.roll(u[..., nu, :, :], -1, mu)
            b = u[..., nu, :, :] @ torch.roll(u[..., mu, :, :], -1, nu)
            tr = (a.real * b.real + a.imag * b.imag).sum((-2, -1)) / nc
            both[0 if mu == 0 else 1] += float((1.0 - tr).sum())
    kin = float((p * p.transpose(-2, -1)).real.sum())
    w = u.reshape(-1, nc, nc)
    w = w @ w.mH - torch.eye(nc, dtype=w.dtype, device="cuda")
    return both[0] + both[1], kin, float((w * w.transpose(-2, -1)).real.sum())


# few blocks, and more than a ticket serves: sites or links in blocks of 256
@pytest.mark.parametrize("nc,dims,precision", [
    (2, [5, 7], "fp64"), (3, [6, 5, 4, 3], "fp32"), (4, [8, 8, 8, 8], "fp64"), (4, [20, 20, 20, 10], "fp64"),
    (4, [24, 24, 24, 16], "fp32"), (3, [24, 24, 26, 26], "fp32"), (3, [24, 24, 24, 24], "fp32-lean"),
    (2, [30, 30, 30, 30], "fp32"), (2, [30, 30, 30, 30], "fp64"), (3, [20, 20, 20, 20], "fp64")])
def test_sums_of_few_and_of_many_blocks(nc, dims, precision):
    with ab.Engine(nc, dims, beta=2.0 * nc, precision=precision, seed=5) as e:
        e.hot_start(3)
        e.initializeE(5, 0)
        u, p = e.get_links(), e.get_momenta(0)
        plaq, kin, _ = torch_sums(u, p, dims, nc)
        for _ in range(2):  # the count of finished blocks starts from zero again
            assert e.EnergyMag() == pytest.approx(plaq, rel=1e-8)
            assert e.simpleenergyEl(0) == pytest.approx(kin, rel=1e-8)
        e.set_links(1.01 * u)
        viol = torch_sums(e.get_links(), p, dims, nc)[2]
        assert e.UViol() == pytest.approx(viol, rel=1e-8)


# slices of fewer elements than threads, of a ragged number, and of several passes
@pytest.mark.parametrize("nc,dims,precision", [(5, [3, 1], "fp64"), (5, [2, 3, 7], "fp32"), (12, [3, 8, 8, 8], "fp64"),
                                               (16, [5, 9, 11], "fp32"), (64, [4, 4, 4, 4], "fp64"), (33, [3, 5, 3], "fp64")])
def test_slice_averages_of_link_major_fields(nc, dims, precision):
    with ab.Engine(nc, dims, beta=2.0 * nc, precision=precision, seed=5) as e:
        e.hot_start(3)
        u = e.get_links().reshape(dims[0], -1, len(dims), nc, nc)[:, :, -1]
        want = np.trace(u, axis1=-2, axis2=-1).real.mean(1) / nc
        np.testing.assert_allclose(e.scalarLoopcorr(), want, rtol=0, atol=1e-12)
