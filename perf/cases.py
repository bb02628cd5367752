"""Performance cases of the engine: what a user of this framework has it do, over the range it is used in.

A case is a dict of plain values.  Its ``kind`` says which public entry points a pass goes through:

``trajectory``  ``Engine.run_trajectories(1, steps)``: one whole HMC trajectory (momentum refresh, H, ``steps``
                fused kick+drift updates, H, Metropolis, accept/reject copy), then the links handed to the
                program's own device buffer with ``Engine.slab_device`` (what a halo exchange or an analysis
                in torch does).  The chain goes on from pass to pass.
``proposal``    the same with the program's own Metropolis test (as the slab chain does): ``loadconfiguration``,
                ``initializeE``, ``hamiltonian``, ``leapfrog``, ``hamiltonian``, the links handed on.  Used for FP32
                storage without residual planes (NC > 4), whose energies are exact enough for a test but not for
                two programs to take every decision alike.
``seam``        one MD step through the reference's own seam, as its main loop calls it:
                ``updateUandcopyDown``, ``updateE``, then the energies, links and momenta read back.
``measure``     the observables of the current configuration: ``measure``, ``scalarLoopcorr``, ``eigenphases``.
``batch``       ``Batch.run``: independent chains of uneven colour number, dimension and volume together,
                ``trajs`` trajectories each, and every chain's links read back.

Links are synthetic: U = exp(i sigma H) with independent Gaussian traceless H and a mean plaquette near that of
a thermalised configuration; momenta are the engine's own Philox draws.  FP32 engines hand their results on in
single precision (complex64 links, float32 energies), FP64 engines in double.  The engines run on their default
kernel mapping (no autotuning), so that a case does the same work on every box.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import askja_b200 as ab

# (colours, extents) of the chains of a batch, taken in turn; small enough for each chain's links to be read back
BATCH_SHAPES = [
    (3, (8, 8, 8, 8)), (2, (16, 16)), (8, (4, 4, 4, 4)), (4, (6, 6, 6)), (3, (5, 7, 9)), (2, (3, 16, 16, 4)),
    (8, (6, 6, 6)), (3, (4, 8, 8, 8)), (5, (5, 6, 7)), (4, (4, 4, 4, 6)), (2, (8, 8, 8)), (6, (4, 4, 4, 4)),
]


def _case(name, kind, nc, dims, steps, prec, level, **more):
    c = {"kind": kind, "nc": nc, "dims": "x".join(str(d) for d in dims), "steps": steps, "prec": prec, "level": level}
    c.update(more)
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest call: one MD step of a small 2-D lattice through the seam functions, where launches count
        _case("seam_su2_24x24_fp64", "seam", 2, (24, 24), 1, "fp64", 6),
        # the reference's CPU-sized production lattice, in its own precision
        _case("traj_su3_8x4_fp64", "trajectory", 3, (8, 8, 8, 8), 50, "fp64", 8),
        # the benchmark's default workload: a full trajectory of a large lattice in FP32
        _case("traj_su3_32x4_fp32", "trajectory", 3, (32, 32, 32, 32), 50, "fp32", 6),
        # the same lattice in FP64 (the benchmark's second leg), a shorter trajectory
        _case("traj_su3_32x4_fp64", "trajectory", 3, (32, 32, 32, 32), 10, "fp64", 6),
        # the benchmark's SU(8) configuration, in both precisions
        _case("hmc_su8_10x4_fp32", "proposal", 8, (10, 10, 10, 10), 20, "fp32", 8),
        _case("traj_su8_10x4_fp64", "trajectory", 8, (10, 10, 10, 10), 20, "fp64", 8),
        # odd colour number, three dimensions, ragged extents (V no multiple of 32)
        _case("traj_su5_17x15x13_fp64", "trajectory", 5, (17, 15, 13), 20, "fp64", 6),
        # the benchmark's SU(16) lattice in FP64: medium colour number
        _case("traj_su16_6x4_fp64", "trajectory", 16, (6, 6, 6, 6), 10, "fp64", 8),
        # the benchmark's SU(32) lattice: large colour number in FP32
        _case("hmc_su32_8x4_fp32", "proposal", 32, (8, 8, 8, 8), 10, "fp32", 8),
        # the largest colour number in FP64, on half of the benchmark's SU(64) lattice
        _case("traj_su64_4x8x16_fp64", "trajectory", 64, (4, 8, 16), 2, "fp64", 8),
        # the observables of a configuration, as the measurement programs take them
        _case("measure_su3_16x4_fp64", "measure", 3, (16, 16, 16, 16), 1, "fp64", 8),
        # a scan of uneven chains advanced together
        _case("batch12_fp32", "batch", 0, (), 20, "fp32", 8, chains=12, trajs=2),
    ]


def draw(rng):
    """One more case of the same ranges: SU(2) to SU(64), two to four dimensions, 100 to a million sites, extents
    odd and even, both precisions, short and long trajectories."""
    kind = rng.choice(["trajectory"] * 6 + ["seam", "measure", "batch"])
    prec = rng.choice(["fp32", "fp64"])
    level = rng.choice([6, 8])
    if kind == "batch":
        return _case(None, kind, 0, (), rng.randint(8, 24), prec, level, chains=rng.randint(3, 12),
                     trajs=rng.randint(1, 2))
    nc = rng.choice([2, 3, 3, 4, 5, 6, 7, 8, 8, 10, 12, 16, 16, 24, 32, 48, 64])
    if kind in ("seam", "measure"):
        nc = min(nc, 16)
    d = rng.choice([2, 3, 4, 4])
    # sites: spread over the logarithm, bounded so that links and matrix products stay below the largest case's
    top = {"trajectory": min(1.0e6, 3.0e7 / (nc * nc * d)), "seam": 4096.0, "measure": min(1.0e5, 4.0e6 / nc ** 3)}[kind]
    if nc > 4:
        top = min(top, 4.0e8 / (nc ** 3 * d))
    vol = math.exp(rng.uniform(math.log(100.0), math.log(max(top, 200.0))))
    side = vol ** (1.0 / d)
    dims = [max(3, int(side * rng.uniform(0.75, 1.3) + 0.5)) for _ in range(d)]
    while np.prod(dims) > max(top, 200.0) and max(dims) > 3:
        dims[dims.index(max(dims))] -= 1
    steps = 1
    if kind == "trajectory":
        room = 8.0e8 if nc > 4 else 5.0e9
        steps = max(1, min(50, int(room / (float(np.prod(dims)) * d * nc ** 3))))
        steps = rng.randint(max(1, steps // 2), steps)
        if prec == "fp32" and nc > 4:
            kind = "proposal"
    return _case(None, kind, nc, dims, steps, prec, level)


# ---- parameters and inputs --------------------------------------------------------------------------------------
def _params(nc):
    beta = 2.0 * nc * nc / (3.0 if nc <= 8 else 1.0)
    return beta, 0.01 if nc <= 8 else 0.004


def _dims(case):
    return [int(d) for d in case["dims"].split("x")] if case["dims"] else []


def _mm(a, b):
    """Product of stacks of square matrices (small ones without a batched GEMM call per matrix)."""
    if a.shape[-1] > 4:
        return torch.matmul(a, b)
    out = a[..., :, 0:1] * b[..., 0:1, :]
    for k in range(1, a.shape[-1]):
        out += a[..., :, k:k + 1] * b[..., k:k + 1, :]
    return out


def _exp(x, order):
    """sum_{k <= order} x^k / k! (Horner)."""
    one = torch.eye(x.shape[-1], dtype=x.dtype, device=x.device)
    e = one + x / order if order else one.expand_as(x).clone()
    for k in range(order - 1, 0, -1):
        e = one + _mm(x, e) / k
    return e


def _links(nc, dims, seed):
    """exp(i sigma H) on every link, [V][D][N][N] complex128 on the GPU (the host layout of the engine)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + nc)
    shape = (int(np.prod(dims)), len(dims), nc, nc)
    h = torch.complex(torch.randn(shape, generator=g, device="cuda", dtype=torch.float64),
                      torch.randn(shape, generator=g, device="cuda", dtype=torch.float64))
    h = 0.5 * (h + h.mH)
    h -= torch.eye(nc, device="cuda", dtype=torch.float64) * (
        h.diagonal(dim1=-2, dim2=-1).real.sum(-1) / nc)[..., None, None]
    u = _exp(h * (0.5j / math.sqrt(nc) / 4), 12)  # |x| < 0.4: the remainder is below rounding
    u = _mm(u, u)
    return _mm(u, u)


def _batch_chains(case, seed):
    out = []
    for i in range(case["chains"]):
        nc, dims = BATCH_SHAPES[i % len(BATCH_SHAPES)]
        beta, dt = _params(nc)
        out.append(dict(nc=nc, dims=list(dims), beta=beta * (1.0 + 0.01 * i), dt=dt, level=case["level"],
                        seed=1000 + 17 * seed + i))
    return out


def _engine(case, seed):
    nc, dims = case["nc"], _dims(case)
    beta, dt = _params(nc)
    e = ab.Engine(nc, dims, beta=beta, dt=dt, level=case["level"], precision=case["prec"], seed=1000 + seed)
    u = _links(nc, dims, seed)
    torch.cuda.synchronize()
    e.slab_device(0, e.vol, u.data_ptr(), False)
    e.takeconfiguration()
    return e, u, dt


def prepare(case, seed):
    if case["kind"] == "batch":
        chains = _batch_chains(case, seed)
        b = ab.Batch(chains, precision=case["prec"])
        for i, c in enumerate(chains):
            b.set_links(i, _links(c["nc"], c["dims"], seed + 31 * i).cpu().numpy())
        return {"case": case, "batch": b}
    e, u, dt = _engine(case, seed)
    if case["kind"] == "seam":
        e.initializeE(1000 + seed, 0)
        e.updateE(0.5 * dt)  # the opening half kick of the reference's main loop
    elif case["kind"] == "measure":
        e.initializeE(1000 + seed, 0)
        e.updateE(0.5 * dt)  # the Gauss law reads the updated momenta
    return {"case": case, "engine": e, "links": u, "dt": dt, "seed": 1000 + seed}


def _single(case, x):
    """What an FP32 engine computed, in single precision."""
    if case["prec"] == "fp64":
        return x
    return np.asarray(x).astype(np.complex64 if np.iscomplexobj(x) else np.float32)


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        res = b.run(case["trajs"], case["steps"])
        return {"h_old": _single(case, np.array([r["h_old"] for r in res])),
                "h_new": _single(case, np.array([r["h_new"] for r in res])),
                "accepted": [int(r["n_acc"]) for r in res],
                "links": [_single(case, b.get_links(i)) for i in range(len(res))]}
    e = state["engine"]
    if case["kind"] == "seam":
        e.updateUandcopyDown(state["dt"])
        e.updateE(state["dt"])
        return {"energies": _single(case, np.array([e.EnergyMag(), e.simpleenergyEl(1)])),
                "links": _single(case, e.get_links()), "momenta": _single(case, e.get_momenta(1))}
    if case["kind"] == "measure":
        w, p = e.eigenphases()
        return {"measure": _single(case, e.measure()), "slices": _single(case, e.scalarLoopcorr()),
                "wilson_phases": _single(case, w), "polyakov_phases": _single(case, p)}
    if case["kind"] == "proposal":
        e.loadconfiguration()
        e.initializeE(state["seed"], 0)
        h_old = e.hamiltonian()
        e.leapfrog(case["steps"], state["dt"])
        out = {"h": _single(case, np.array([h_old, e.hamiltonian()]))}
    else:
        r, _ = e.run_trajectories(1, case["steps"], want_log=False)
        out = {"h": _single(case, np.array([r["h_old"], r["h_new"]])), "accepted": int(r["accepted"] != 0)}
    u = state["links"]
    e.slab_device(0, e.vol, u.data_ptr(), True)
    if case["prec"] != "fp64":
        with torch.cuda.stream(torch.cuda.ExternalStream(e.stream_ptr)):
            u = u.to(torch.complex64)
    return {**out, "links": u}


# ---- what a pass cannot do without --------------------------------------------------------------------------------
def _md_work(nc, dims, steps, prec):
    """Bytes and flops of `steps` MD steps: links and momenta read and written once per step; 4(D-1) staple
    products, the product with the link and four for the exponential."""
    links = float(np.prod(dims)) * len(dims)
    size = 8 if prec == "fp32" else 16
    return links * steps * 4 * nc * nc * size, links * steps * (4 * (len(dims) - 1) + 5) * 8.0 * nc ** 3


def work(case):
    if case["kind"] == "batch":
        both = [_md_work(c["nc"], c["dims"], case["steps"] * case["trajs"], case["prec"])
                for c in _batch_chains(case, 0)]
        return {"bytes": sum(b for b, _ in both), "flops": sum(f for _, f in both)}
    nc, dims = case["nc"], _dims(case)
    if case["kind"] == "measure":  # links and momenta read once; two products a plaquette, two a link for Gauss
        links = float(np.prod(dims)) * len(dims)
        planes = len(dims) * (len(dims) - 1) / 2
        return {"bytes": links * 2 * nc * nc * (8 if case["prec"] == "fp32" else 16),
                "flops": 8.0 * nc ** 3 * (2 * planes * float(np.prod(dims)) + 3 * links)}
    b, f = _md_work(nc, dims, case["steps"], case["prec"])
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits, in plain torch ----------------------------------------------------------------------------
def _philox(ctr, key):
    """Philox4x32-10 on int64 tensors (Salmon, Moraes, Dror, Shaw, SC'11): ctr four tensors, key two words."""
    m = 0xFFFFFFFF
    x, y, z, w = ctr
    k0, k1 = key
    for _ in range(10):
        p0, p1 = x * 0xD2511F53, z * 0xCD9E8D57
        x, y, z, w = ((p1 >> 32) & m) ^ y ^ k0, p1 & m, ((p0 >> 32) & m) ^ w ^ k1, p0 & m
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    return x, y, z, w


def _u01(w):
    return (w.double() + 0.5) / 4294967296.0


def _momenta(nc, vol, d, seed, traj, beta):
    """The refresh: P = sqrt(2N/beta) sum_a xi_a T_a, normals by Box-Muller from blocks (a/4, link, 0, traj)."""
    key = (seed & 0xFFFFFFFF, seed >> 32)
    link = torch.arange(vol * d, device="cuda")
    zero = torch.zeros_like(link)
    xi = []
    for blk in range((nc * nc - 1 + 3) // 4):
        x, y, z, w = (_u01(v) for v in _philox((zero + blk, link & 0xFFFFFFFF, link >> 32, zero + traj), key))
        for r, t in ((x, y), (z, w)):
            rad = torch.sqrt(-2.0 * torch.log(r))
            xi += [rad * torch.cos(2 * math.pi * t), rad * torch.sin(2 * math.pi * t)]
    p = torch.zeros((vol * d, nc, nc), dtype=torch.complex128, device="cuda")
    a = 0
    for i in range(nc):
        for j in range(i + 1, nc):
            p[:, i, j] = torch.complex(0.5 * xi[a], -0.5 * xi[a + 1])
            p[:, j, i] = torch.complex(0.5 * xi[a], 0.5 * xi[a + 1])
            a += 2
    for m in range(nc - 1):
        nm = math.sqrt(0.5 / ((m + 1) * (m + 2)))
        for k in range(m + 1):
            p[:, k, k] += nm * xi[a + m]
        p[:, m + 1, m + 1] -= (m + 1) * nm * xi[a + m]
    p *= math.sqrt(2.0 * nc / beta)
    return [p.view(vol, d, nc, nc)[:, k].clone() for k in range(d)]


def _force(u, dims):
    """Adjoint(U_mu sum of staples) of every link; u: one [V][N][N] stack per direction."""
    d, nc = len(dims), u[0].shape[-1]

    def at(x, step, axis):  # the stack at x + step e_axis
        return torch.roll(x.view(*dims, nc, nc), -step, axis).reshape(-1, nc, nc)

    out = []
    for mu in range(d):
        s = torch.zeros_like(u[mu])
        for nu in range(d):
            if nu == mu:
                continue
            far = at(u[nu], 1, mu)
            s += _mm(_mm(far, at(u[mu], 1, nu).mH), u[nu].mH)
            s += at(_mm(_mm(u[mu], far).mH, u[nu]), -1, nu)
        w = _mm(u[mu], s)
        w = w - w.mH
        tr = w.diagonal(dim1=-2, dim2=-1).sum(-1) / nc
        w.diagonal(dim1=-2, dim2=-1).sub_(tr[:, None])
        out.append(-0.5j * w)
    return out


def _plaquettes(u, dims):
    """Temporal and spatial sums of 1 - ReTr P / N."""
    d, nc = len(dims), u[0].shape[-1]
    both = [0.0, 0.0]
    for mu in range(d):
        for nu in range(mu + 1, d):
            a = _mm(u[mu], torch.roll(u[nu].view(*dims, nc, nc), -1, mu).reshape(-1, nc, nc))
            b = _mm(u[nu], torch.roll(u[mu].view(*dims, nc, nc), -1, nu).reshape(-1, nc, nc))
            tr = (a.real * b.real + a.imag * b.imag).sum((-2, -1)) / nc
            both[0 if mu == 0 else 1] += float((1.0 - tr).sum())
    return both


def _tr2(p):
    return sum(float((x * x.transpose(-2, -1)).real.sum()) for x in p)


def _kick(u, p, eps, dims):
    for x, f in zip(p, _force(u, dims)):
        x -= eps * f


def _drift(u, p, eps, order):
    return [_mm(_exp((1j * eps) * x, order), y) for x, y in zip(p, u)]


def _exact_trajectory(u, dims, beta, dt, level, steps, seed, traj, test=True):
    nc = u[0].shape[-1]
    p = _momenta(nc, int(np.prod(dims)), len(dims), seed, traj, beta)
    h_old = beta * (sum(_plaquettes(u, dims)) + _tr2(p) / (2 * nc))
    v = u
    for k in range(steps):
        _kick(v, p, 0.5 * dt if k == 0 else dt, dims)
        v = _drift(v, p, dt, level)
    _kick(v, p, 0.5 * dt, dims)
    h_new = beta * (sum(_plaquettes(v, dims)) + _tr2(p) / (2 * nc))
    words = _philox([torch.tensor([c]) for c in (0xFFFFFFFF, 0, 0, traj)], (seed & 0xFFFFFFFF, seed >> 32))
    accept = h_new < h_old or float(_u01(words[0])) < math.exp(h_old - h_new)
    return h_old, h_new, v if accept or not test else u


def _closed_lines(u, dims, axis, along):
    """Matrices of the closed lines along `axis` through the sites of the `along` axis (the others 0)."""
    nc = u[0].shape[-1]
    x = u[axis].view(*dims, nc, nc)
    for a in reversed(range(len(dims))):
        if a not in (axis, along):
            x = x.select(a, 0)
    if axis < along:
        x = x.transpose(0, 1)
    w = x[:, 0]
    for k in range(1, dims[axis]):
        w = torch.matmul(w, x[:, k])
    return w


def _mean_phases(w):
    nc = w.shape[-1]
    ph = np.angle(np.linalg.eigvals(w.cpu().numpy()))
    wind = ph.sum(1) / (2 * math.pi)
    ph -= np.where(np.abs(wind) > 0.1, wind * 2 * math.pi / nc, 0.0)[:, None]
    return np.sort(ph, axis=1).mean(0)


def _exact_measure(u, p, dims):
    d, nc = len(dims), u[0].shape[-1]

    def mean_line(axis, along):
        w = _closed_lines(u, dims, axis, along)
        return float(w.diagonal(dim1=-2, dim2=-1).sum(-1).abs().mean()) / nc

    gauss = sum((x - _mm(_mm(y.mH, x), y)).sum(0) for x, y in zip(p, u))
    one = torch.eye(nc, dtype=torch.complex128, device="cuda")
    out = _plaquettes(u, dims) + [mean_line(0, 1)] + [mean_line(k, 0) for k in range(1, d)]
    out += [float((gauss * gauss.T).real.sum()), _tr2([_mm(y, y.mH) - one for y in u])]
    tr = u[d - 1].diagonal(dim1=-2, dim2=-1).real.sum(-1) / nc
    return {"measure": np.array(out), "slices": tr.view(dims[0], -1).mean(1).cpu().numpy(),
            "wilson_phases": _mean_phases(_closed_lines(u, dims, 1, 0)),
            "polyakov_phases": _mean_phases(_closed_lines(u, dims, 0, 1))}


def _whole(u):
    return torch.stack(u, 1)


def exact(case, seed):
    level = case["level"]
    if case["kind"] == "batch":
        h, links = [], []
        for i, c in enumerate(_batch_chains(case, seed)):
            x = _links(c["nc"], c["dims"], seed + 31 * i)
            u = [x[:, k].clone() for k in range(len(c["dims"]))]
            for t in range(case["trajs"]):
                h_old, h_new, u = _exact_trajectory(u, c["dims"], c["beta"], c["dt"], level, case["steps"], c["seed"], t)
            h.append((h_old, h_new))
            links.append(_whole(u))
        h = np.array(h)
        return {"h_old": h[:, 0].copy(), "h_new": h[:, 1].copy(), "links": links}
    nc, dims = case["nc"], _dims(case)
    if nc >= 16 and case["steps"] * np.prod(dims) * len(dims) * nc ** 3 > 8.0e9:
        return None
    beta, dt = _params(nc)
    x = _links(nc, dims, seed)
    u = [x[:, k].clone() for k in range(len(dims))]
    del x
    if case["kind"] in ("trajectory", "proposal"):
        h_old, h_new, u = _exact_trajectory(u, dims, beta, dt, level, case["steps"], 1000 + seed, 0,
                                            case["kind"] == "trajectory")
        return {"h": np.array([h_old, h_new]), "links": _whole(u)}
    p = _momenta(nc, int(np.prod(dims)), len(dims), 1000 + seed, 0, beta)
    _kick(u, p, 0.5 * dt, dims)
    if case["kind"] == "measure":
        return _exact_measure(u, p, dims)
    u = _drift(u, p, dt, level)
    _kick(u, p, dt, dims)
    return {"energies": np.array([sum(_plaquettes(u, dims)), _tr2(p)]), "links": _whole(u), "momenta": _whole(p)}
