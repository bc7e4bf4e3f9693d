"""Performance cases: what a user of this package has it do, over its real sizes.

Every case goes through the package's public classes and functions as a
program would call them:

  sim      ``ChLLSim.run`` on host arrays (the reference's own class: upload,
           sweeps with measurement rows, download)
  sweep    a device-resident ``Lattice``: sweeps, one FP64 measurement, the
           state back in natural order on the device
  anneal   ``workflows.anneal``: temperature stages with rows every few sweeps
  batch    ``Batch.run`` over a phase grid of uneven lattices, the moments and
           two configurations read back
  grid     ``workflows.phase_diagram``: the whole call, from specs to summaries
           (creation, launch-shape tuning, sweeps, moments)
  energy   ``lattice_energy`` forward and backward (torch autograd)
  torque   ``tangent_gradient`` and ``coupling_sensitivities``
  quench   ``autograd.quench`` of a configuration, its energies and end state
  measure  a configuration on the device loaded and observed (FP64 row)
  shells   ``shell_correlations`` of a configuration
  stripes  ``structure_factor`` along a lattice direction

A case is a dict of plain values; ``listed()`` names twelve of them and
``draw(rng)`` gives more of the same ranges.  ``prepare`` makes inputs from the
seed alone, ``run`` is one pass, ``work`` the bytes and operations a pass cannot
do without, and ``exact`` what it returns in 64 bits where that has a value of
its own: a Metropolis chain has none (every accept decision is a comparison
with a random number), so the chain cases return None there.
"""
import math

import numpy as np
import torch

# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------


def _shape(ni, nj=None, nk=None):
    return {"ni": ni, "nj": ni if nj is None else nj, "nk": ni if nk is None else nk}


def listed():
    return [
        # The reference's own small case, as its driver scripts run it: one
        # ChLLSim, 1000 sweeps, a row every 100.
        dict(name="sim_32", kind="sim", **_shape(32), boundary="periodic", kT=0.5, K=0.5, g=0.0,
             sweeps=1000, every=100),
        # The 128^3 anneal: two of its temperature stages, rows every 10 sweeps
        # (a mid-size lattice that fits in L2).
        dict(name="anneal_128", kind="anneal", **_shape(128), boundary="periodic", kT=0.8,
             kT_end=0.7, K=1.0, g=0.25, stages=2, sweeps=100, every=10),
        # The large lattice: 480^3, sweeps bound by HBM, then a measurement and
        # the configuration handed to the caller.
        dict(name="sweep_480", kind="sweep", **_shape(480), boundary="periodic", kT=0.3, K=1.0,
             g=0.0, sweeps=20),
        # The reference's default boundary (open) on odd, unequal edges whose
        # rows need padding.
        dict(name="sweep_ragged", kind="sweep", **_shape(150, 125, 101), boundary="open", kT=0.6,
             K=1.0, g=0.1, sweeps=50),
        # A phase diagram of 64 uneven replicas with measurements every 50
        # sweeps, as the reference's phase-diagram driver measures.
        dict(name="batch_grid", kind="batch", nkT=8, ng=8, sizes="32,48,64", sweeps=200, every=50),
        # The whole phase-diagram call for a 4 x 4 grid of one size.
        dict(name="phase_diagram", kind="grid", nkT=4, ng=4, size=48, sweeps=500, every=50),
        # The differentiation workload: energy and gradients of a 64^3 lattice
        # (a latency-bound call inside an optimisation loop).
        dict(name="energy_64", kind="energy", **_shape(64), boundary="periodic", K=1.0, h=0.5,
             eps=1.0),
        # Torques and coupling sensitivities of a large, ragged, open lattice.
        dict(name="torque_ragged", kind="torque", **_shape(250, 181, 129), boundary="open", K=0.8,
             h=0.3, eps=1.2),
        # The zero-temperature quench of the differentiation workload.
        dict(name="quench_64", kind="quench", **_shape(64), boundary="periodic", K=1.0, h=0.5,
             eps=1.0, eta=0.05, steps=200, report=100),
        # Analysing a configuration: load it and take the FP64 observables.
        dict(name="measure_256", kind="measure", **_shape(256), boundary="periodic", K=1.0, h=0.5,
             eps=1.0),
        # Shell correlations out to ten sites, open as in the reference notebook.
        dict(name="shells_96", kind="shells", **_shape(96), boundary="open", shells=10,
             wrap=False),
        # The chirality structure factor over 500 wave numbers along [1, 1, 1].
        dict(name="stripes_256", kind="stripes", **_shape(256), boundary="open", bins=500, px=1,
             py=1, pz=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_shape(rng, lo, hi, boundary):
    """Three edges around one size of [lo, hi] (log-uniform), even where the
    boundary is periodic."""
    base = _log_int(rng, lo, hi)
    edges = [min(hi, max(lo, int(round(base * rng.uniform(0.7, 1.3))))) for _ in range(3)]
    if boundary == "periodic":
        edges = [e - e % 2 for e in edges]
    return _shape(*edges)


def draw(rng):
    kind = rng.choice(["sim", "sweep", "sweep", "anneal", "batch", "grid", "energy", "energy",
                       "torque", "quench", "measure", "measure", "shells", "stripes"])
    boundary = rng.choice(["periodic", "open"])
    kT, K = round(rng.uniform(0.1, 1.5), 3), round(rng.uniform(0.2, 1.2), 3)
    g, eps = round(rng.uniform(0.0, 0.6), 3), round(rng.uniform(0.8, 1.3), 3)
    if kind == "sim":
        every = rng.choice([20, 50, 100])
        return dict(kind=kind, **_draw_shape(rng, 10, 96, boundary), boundary=boundary, kT=kT, K=K,
                    g=g, sweeps=every * rng.randint(2, 6), every=every)
    if kind == "sweep":
        return dict(kind=kind, **_draw_shape(rng, 8, 400, boundary), boundary=boundary, kT=kT, K=K,
                    g=g, sweeps=rng.randint(1, 20))
    if kind == "anneal":
        return dict(kind=kind, **_draw_shape(rng, 16, 160, boundary), boundary=boundary, kT=kT,
                    kT_end=round(0.8 * kT, 4), K=K, g=g, stages=2,
                    sweeps=10 * rng.randint(2, 10), every=10)
    if kind == "batch":
        return dict(kind=kind, nkT=rng.randint(2, 8), ng=rng.randint(2, 8),
                    sizes=",".join(str(2 * rng.randint(8, 32)) for _ in range(3)),
                    sweeps=10 * rng.randint(4, 15), every=rng.choice([10, 20, 50]))
    if kind == "grid":
        return dict(kind=kind, nkT=rng.randint(2, 6), ng=rng.randint(1, 6),
                    size=2 * rng.randint(8, 32), sweeps=10 * rng.randint(10, 50),
                    every=rng.choice([10, 50]))
    if kind == "energy":
        return dict(kind=kind, **_draw_shape(rng, 8, 256, boundary), boundary=boundary, K=K, h=g,
                    eps=eps)
    if kind == "torque":
        return dict(kind=kind, **_draw_shape(rng, 16, 256, boundary), boundary=boundary, K=K, h=g,
                    eps=eps)
    if kind == "quench":
        return dict(kind=kind, **_draw_shape(rng, 12, 128, boundary), boundary=boundary, K=K, h=g,
                    eps=eps, eta=0.05, steps=rng.randint(20, 100), report=rng.choice([10, 50]))
    if kind == "measure":
        return dict(kind=kind, **_draw_shape(rng, 8, 400, boundary), boundary=boundary, K=K, h=g,
                    eps=eps)
    if kind == "shells":
        shells = rng.randint(3, 12)
        wrap = boundary == "periodic"
        return dict(kind=kind, **_draw_shape(rng, 2 * shells, 112, boundary), boundary=boundary,
                    shells=shells, wrap=wrap)
    px, py, pz = rng.choice([(1, 1, 1), (1, 0, 0), (0, 0, 1), (1, 1, 0), (1, -1, 2)])
    return dict(kind=kind, **_draw_shape(rng, 16, 320, boundary), boundary=boundary,
                bins=rng.randint(50, 600), px=px, py=py, pz=pz)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------


def _dims(case):
    return case["ni"], case["nj"], case["nk"]


def _sites(case):
    return case["ni"] * case["nj"] * case["nk"]


def _configuration(case, seed):
    """A cholesteric configuration with thermal noise, (N, 4) FP32 in natural
    order (i fastest): directors that twist along z, chiralities in stripes."""
    ni, nj, nk = _dims(case)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    a = torch.randn((nk, nj, ni, 3), generator=gen, device="cuda", dtype=torch.float32).mul_(0.25)
    u = torch.rand((nk, nj, ni), generator=gen, device="cuda", dtype=torch.float32)
    start = torch.rand(2, generator=gen, device="cuda", dtype=torch.float32)
    z = torch.arange(nk, device="cuda", dtype=torch.float32).view(nk, 1, 1)
    y = torch.arange(nj, device="cuda", dtype=torch.float32).view(1, nj, 1)
    x = torch.arange(ni, device="cuda", dtype=torch.float32).view(1, 1, ni)
    twist = 6.2831853 * (z / 20.0 + start[0])
    a[..., 0] += torch.cos(twist)
    a[..., 1] += torch.sin(twist)
    a /= a.norm(dim=-1, keepdim=True)
    stripes = 0.5 + 0.45 * torch.sin(6.2831853 * ((x + y + z) / 24.0 + start[1]))
    out = torch.empty((nk, nj, ni, 4), device="cuda", dtype=torch.float32)
    out[..., :3] = a
    out[..., 3] = torch.where(u < stripes, 1.0, -1.0)
    return out.view(-1, 4)


def _grid_axes(case):
    return np.linspace(0.1, 2.0, case["nkT"]), np.linspace(0.0, 3.0, case["ng"])


def prepare(case, seed):
    from chllmodel_b200.lattice import Lattice, coupling

    kind = case["kind"]
    st = {"case": case, "seed": int(seed)}
    if kind == "sim":
        from chllmodel_b200.chll import ChLLSim

        rng = np.random.default_rng(seed)
        sim = ChLLSim(*_dims(case), case["kT"], 0.1, case["K"], case["g"], 0.0, seed=int(seed),
                      boundary=case["boundary"], verbose=False)
        sim.init_random_directors(rng)
        sim.init_with_s(np.where(rng.random(_dims(case)) < 0.5, -1, 1))
        st["sim"] = sim
        return st
    if kind == "batch":
        from chllmodel_b200.batched import Batch, phase_grid

        kTs, gs = _grid_axes(case)
        sizes = [int(v) for v in case["sizes"].split(",")]
        st["batch"] = Batch(phase_grid(kTs, gs, sizes, K=1.0, seed=int(seed), size_seed=12345))
        st["batch"].init_random()
        return st
    if kind == "grid":
        return st
    if kind in ("energy", "torque"):
        state = _configuration(case, seed)
        st["n"] = state[:, :3].contiguous()
        st["s"] = state[:, 3].contiguous()
        if kind == "energy":
            st["n"].requires_grad_(True)
            for name in ("eps", "K", "h"):
                st[name] = torch.tensor(float(case[name]), dtype=torch.float64,
                                        requires_grad=True)
        return st
    lat = st["lat"] = Lattice(*_dims(case), boundary=case["boundary"])
    if kind in ("sweep", "anneal"):
        lat.init_random(int(seed))
        lat.set_control(0.1, step=1)
        st["out"] = torch.empty((lat.nsites, 4), dtype=torch.float32, device="cuda")
        if kind == "sweep":
            st["cp"] = coupling(case["kT"], case["K"], case["g"])
        return st
    state = _configuration(case, seed)
    torch.cuda.synchronize()
    if kind in ("quench", "measure"):
        st["state"] = state
        st["out"] = torch.empty_like(state) if kind == "quench" else None
        if kind == "measure":
            st["cp"] = coupling(0.0, case["K"], case["h"], case["eps"])
    else:  # shells, stripes: the lattice holds the configuration
        lat.upload_f4(state.data_ptr())
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------


def _columns(records):
    """A list of dicts of numbers as one array per field."""
    return {k: np.array([r[k] for r in records], dtype=np.float64)
            for k in records[0] if isinstance(records[0][k], (int, float))}


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "sim":
        sim = st["sim"]
        sim.run(case["sweeps"], case["every"])
        return {"nx": sim.nx, "ny": sim.ny, "nz": sim.nz, "s": sim.s, "m": sim.m,
                "msteps": sim.msteps, "rows": sim.rows, "d": float(sim.d)}
    if kind == "sweep":
        lat = st["lat"]
        lat.sweep(st["cp"], case["sweeps"], seed=st["seed"])
        row = lat.observe(st["cp"])
        lat.download_f4(st["out"].data_ptr())
        return {"row": row, "state": st["out"]}
    if kind == "anneal":
        from chllmodel_b200.workflows import anneal, linear_schedule

        lat = st["lat"]
        stages = anneal(lat, linear_schedule(case["kT"], case["kT_end"], case["stages"]),
                        case["sweeps"], K=case["K"], g=case["g"], seed=st["seed"],
                        measure_every=case["every"])
        lat.download_f4(st["out"].data_ptr())
        return {"stages": _columns(stages), "state": st["out"]}
    if kind == "batch":
        b = st["batch"]
        b.run(case["sweeps"], case["every"])
        m = b.moments()
        return {"moments": m, "first": b.download_f4(0), "last": b.download_f4(len(b) - 1)}
    if kind == "grid":
        from chllmodel_b200.workflows import phase_diagram

        kTs, gs = _grid_axes(case)
        return _columns(phase_diagram(kTs, gs, [case["size"]], K=1.0, nsweeps=case["sweeps"],
                                      measure_every=case["every"], seed=st["seed"]))
    if kind == "energy":
        from chllmodel_b200.autograd import lattice_energy

        E = lattice_energy(st["n"], st["s"], st["eps"], st["K"], st["h"], _dims(case),
                           case["boundary"])
        gn, ge, gk, gh = torch.autograd.grad(E, [st["n"], st["eps"], st["K"], st["h"]])
        return {"E": E.detach(), "dn": gn, "deps": ge, "dK": gk, "dh": gh}
    if kind == "torque":
        from chllmodel_b200.autograd import coupling_sensitivities, tangent_gradient

        args = (st["n"], st["s"], case["eps"], case["K"], case["h"], _dims(case), case["boundary"])
        t = tangent_gradient(*args)
        return {"torque": t, **{k: float(v) for k, v in coupling_sensitivities(*args).items()}}
    lat = st["lat"]
    if kind == "quench":
        from chllmodel_b200.autograd import quench

        lat.upload_f4(st["state"].data_ptr())
        energies = quench(lat, case["eps"], case["K"], case["h"], case["eta"], case["steps"],
                          report_every=case["report"])
        lat.download_f4(st["out"].data_ptr())
        return {"steps": np.array([s for s, _ in energies]),
                "energies": np.array([e for _, e in energies]), "state": st["out"]}
    if kind == "measure":
        lat.upload_f4(st["state"].data_ptr())
        return {"row": lat.observe(st["cp"])}
    if kind == "shells":
        from chllmodel_b200.analysis import shell_correlations

        gn, gs, counts = shell_correlations(lat, case["shells"], wrap=case["wrap"])
        return {"gn": gn, "gs": gs, "counts": counts}
    from chllmodel_b200.analysis import structure_factor

    sf, kvs = structure_factor(lat, case["bins"], 0.0, 0.5, [case["px"], case["py"], case["pz"]])
    return {"sf": sf, "kvs": kvs}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

# A sweep reads every site (16 B) in each colour's pass and writes it once:
# 48 B per site.  Operations of a site's trials: two sets of six bond sums (18
# each), the proposal, two acceptances.
_SWEEP_BYTES, _SWEEP_FLOPS = 48, 270
_MEASURE_BYTES, _MEASURE_FLOPS = 16, 75
_GRAD_FLOPS = 6 * 30 + 3 * 16


def _grid_sites(case):
    from chllmodel_b200.batched import phase_grid

    kTs, gs = _grid_axes(case)
    sizes = [int(v) for v in case["sizes"].split(",")] if "sizes" in case else [case["size"]]
    return sum(sp["ni"] ** 3 for sp in phase_grid(kTs, gs, sizes, size_seed=12345))


def _shell_pairs(case):
    """Unordered pairs of sites within the shells (each site with itself once)."""
    R, n = case["shells"], _dims(case)
    d = np.arange(-R + 1, R)
    dx, dy, dz = np.meshgrid(d, d, d, indexing="ij")
    inside = dx * dx + dy * dy + dz * dz < R * R
    if case["wrap"]:
        total = float(inside.sum()) * _sites(case)
    else:
        w = (np.clip(n[0] - abs(dx), 0, None) * np.clip(n[1] - abs(dy), 0, None) *
             np.clip(n[2] - abs(dz), 0, None))
        total = float(w[inside].sum())
    return (total + _sites(case)) / 2


def work(case):
    kind = case["kind"]
    if kind in ("batch", "grid"):
        n, sw = _grid_sites(case), case["sweeps"]
        meas = sw // case["every"]
        return {"bytes": n * (_SWEEP_BYTES * sw + _MEASURE_BYTES * meas),
                "flops": n * (_SWEEP_FLOPS * sw + _MEASURE_FLOPS * meas)}
    n = _sites(case)
    if kind == "sim":
        meas, sw = case["sweeps"] // case["every"], case["sweeps"]
        return {"bytes": n * (_SWEEP_BYTES * sw + _MEASURE_BYTES * meas + 2 * 28),
                "flops": n * (_SWEEP_FLOPS * sw + _MEASURE_FLOPS * meas)}
    if kind == "sweep":
        return {"bytes": n * (_SWEEP_BYTES * case["sweeps"] + _MEASURE_BYTES + 32),
                "flops": n * (_SWEEP_FLOPS * case["sweeps"] + _MEASURE_FLOPS)}
    if kind == "anneal":
        sw = case["stages"] * case["sweeps"]
        meas = sw // case["every"]
        return {"bytes": n * (_SWEEP_BYTES * sw + _MEASURE_BYTES * meas + 32),
                "flops": n * (_SWEEP_FLOPS * sw + _MEASURE_FLOPS * meas)}
    if kind == "energy":  # directors and chiralities in, the gradient out
        return {"bytes": n * (16 + 12), "flops": n * _GRAD_FLOPS}
    if kind == "torque":  # two calls: directors and chiralities in twice, the torque out
        return {"bytes": n * (16 + 12 + 16), "flops": n * (_GRAD_FLOPS + 3 * 16 + 20)}
    if kind == "quench":  # two colour passes of 24 B per site and step
        reports = -(-case["steps"] // case["report"])
        return {"bytes": n * (48 * case["steps"] + 16 * reports + 64),
                "flops": n * (200 * case["steps"] + 48 * reports)}
    if kind == "measure":
        return {"bytes": n * 16, "flops": n * _MEASURE_FLOPS}
    if kind == "shells":
        return {"bytes": n * 16, "flops": 9 * _shell_pairs(case)}
    p = [abs(case[k]) for k in ("px", "py", "pz")]
    planes = sum(a * d for a, d in zip(p, _dims(case)))
    return {"bytes": n * 16, "flops": n * 4 + 10.0 * case["bins"] * planes}


# ---------------------------------------------------------------------------
# The same in 64 bits, by plain torch
# ---------------------------------------------------------------------------

# (nk, nj, ni) grids: axis 0, 1, 2 of the lattice (x, y, z) is dimension 2, 1, 0
_DIM = (2, 1, 0)


def _cross(n, b, axis):
    """(n x b) . e_axis"""
    p, q = (axis + 1) % 3, (axis + 2) % 3
    return n[..., p] * b[..., q] - n[..., q] * b[..., p]


def _split(case, state):
    ni, nj, nk = _dims(case)
    grid = state.double().view(nk, nj, ni, 4)
    return grid[..., :3].clone(), grid[..., 3].clone()


def _energy64(n, s, eps, K, h, periodic):
    """Total energy, each bond once."""
    total = -h * s.sum()
    for axis, dim in enumerate(_DIM):
        m, L = n, n.shape[dim]
        b, sb, sm = torch.roll(n, -1, dim), torch.roll(s, -1, dim), s
        if not periodic:
            m, b = m.narrow(dim, 0, L - 1), b.narrow(dim, 0, L - 1)
            sm, sb = sm.narrow(dim, 0, L - 1), sb.narrow(dim, 0, L - 1)
        c = (m * b).sum(-1)
        total = total + (eps * (1.0 - c * c) - K * c * _cross(m, b, axis) * 0.5 * (sm + sb)).sum()
    return total


def _gradient64(case, state):
    """E, dE/dn, dE/d(eps, K, h) by automatic differentiation."""
    n, s = _split(case, state)
    n.requires_grad_(True)
    c = [torch.tensor(float(case[k]), dtype=torch.float64, device="cuda", requires_grad=True)
         for k in ("eps", "K", "h")]
    E = _energy64(n, s, *c, case["boundary"] == "periodic")
    return (n.detach(), E.detach()) + torch.autograd.grad(E, [n] + c)


def _tangent(n, g):
    return g - (g * n).sum(-1, keepdim=True) * n / (n * n).sum(-1, keepdim=True)


def _row64(case, state):
    """The measurement row of a configuration just loaded."""
    n, s = _split(case, state)
    eps, K, h = case["eps"], case["K"], case["h"]
    N = float(s.numel())
    E = _energy64(n, s, eps, K, h, case["boundary"] == "periodic")
    # the reference's etot(): x and y periodic, z open, and the x component of
    # the +y neighbour in the dot product read from the +x +y neighbour
    ref = -h * s.sum()
    for axis, dim in enumerate(_DIM):
        b, sb = torch.roll(n, -1, dim), torch.roll(s, -1, dim)
        d = b
        if axis == 1:
            d = b.clone()
            d[..., 0] = torch.roll(b[..., 0], -1, 2)
        c = (n * d).sum(-1)
        t = eps * (1.0 - c * c) - K * c * _cross(n, b, axis) * 0.5 * (s + sb)
        ref = ref + (t[:-1].sum() if axis == 2 else t.sum())
    q = [(n[..., i] * n[..., j]).sum() for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
    E, ref, ss = float(E), float(ref), float(s.sum())
    return np.array([ref / N, ss / N, 0.0, 0.0, 0.1, E, ss] + [float(v) for v in q] +
                    [ref, 0.0, N])


def _quench64(case, state):
    n, s = _split(case, state)
    eps, K, h, eta = (case[k] for k in ("eps", "K", "h", "eta"))
    periodic = case["boundary"] == "periodic"
    ni, nj, nk = _dims(case)
    z, y, x = torch.meshgrid(*(torch.arange(v, device="cuda") for v in (nk, nj, ni)),
                             indexing="ij")
    colour = ((x + y + z) % 2).unsqueeze(-1)
    edge = {}
    for dim, pos in zip((2, 1, 0), (x, y, z)):
        L = n.shape[dim]
        edge[dim] = ((pos < L - 1).double(), (pos > 0).double())

    def gradient():
        g = torch.zeros_like(n)
        for axis, dim in enumerate(_DIM):
            p, q = (axis + 1) % 3, (axis + 2) % 3
            for which, (shift, sigma) in enumerate(((-1, -1.0), (1, 1.0))):
                b = torch.roll(n, shift, dim)
                sbar = 0.5 * (s + torch.roll(s, shift, dim))
                c, X = (n * b).sum(-1), _cross(n, b, axis)
                w = sigma * K * sbar
                t = (-2.0 * eps * c + w * X).unsqueeze(-1) * b
                t[..., p] += w * c * b[..., q]
                t[..., q] -= w * c * b[..., p]
                g += t if periodic else t * edge[dim][which].unsqueeze(-1)
        return g

    energies = []
    for step in range(1, case["steps"] + 1):
        for col in (0, 1):
            m = n - eta * _tangent(n, gradient())
            n = torch.where(colour == col, m / m.norm(dim=-1, keepdim=True), n)
        if step % case["report"] == 0 or step == case["steps"]:
            energies.append(float(_energy64(n, s, eps, K, h, periodic)))
    return {"steps": None, "energies": np.array(energies),
            "state": torch.cat([n, s.unsqueeze(-1)], -1).view(-1, 4)}


def _shells64(case, state):
    n, s = _split(case, state)
    R = case["shells"]
    lens = n.shape[:3]
    sums = torch.zeros((2, R), dtype=torch.float64, device="cuda")
    counts = np.zeros(R)
    d = range(-R + 1, R)
    for dk in d:
        for dj in d:
            for di in d:
                r2 = di * di + dj * dj + dk * dk
                half = dk > 0 or (dk == 0 and (dj > 0 or (dj == 0 and di >= 0)))
                if r2 >= R * R or not half:
                    continue
                shell = math.isqrt(r2)
                weight = 1.0 if r2 == 0 else 2.0
                if case["wrap"]:
                    b, t = (torch.roll(v, (-dk, -dj, -di), (0, 1, 2)) for v in (n, s))
                    a, u = n, s
                else:
                    if any(abs(o) >= L for o, L in zip((dk, dj, di), lens)):
                        continue
                    here = tuple(slice(max(0, -o), L - max(0, o)) for o, L in zip((dk, dj, di), lens))
                    there = tuple(slice(max(0, o), L - max(0, -o)) for o, L in zip((dk, dj, di), lens))
                    a, b, u, t = n[here], n[there], s[here], s[there]
                c = (a * b).sum(-1)
                sums[0, shell] += weight * (c * c).sum()
                sums[1, shell] += weight * (u * t).sum()
                counts[shell] += weight * c.numel()
    mean = float(s.mean())
    gn, gs = sums.cpu().numpy() / counts
    return {"gn": gn, "gs": gs - mean * mean, "counts": counts}


def _stripes64(case, state):
    _, s = _split(case, state)
    kvs = np.linspace(0.0, 0.5, case["bins"])
    k = torch.from_numpy(kvs).cuda()
    sc = torch.zeros(len(kvs), dtype=torch.complex128, device="cuda")
    waves = []
    for p, L in zip((case["px"], case["py"], case["pz"]), _dims(case)):
        ph = torch.outer(p * torch.arange(1, L + 1, device="cuda", dtype=torch.float64), k)
        waves.append(torch.polar(torch.ones_like(ph), -ph))
    for plane in range(s.shape[0]):
        rows = torch.complex(s[plane] @ waves[0].real, s[plane] @ waves[0].imag)  # (nj, bins)
        sc += (rows * waves[1]).sum(0) * waves[2][plane]
    sc = sc.cpu().numpy() / s.numel()
    return {"sf": sc.real ** 2 + sc.imag ** 2, "kvs": kvs}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sim", "sweep", "anneal", "batch", "grid"):
        return None
    state = _configuration(case, seed)
    if kind in ("energy", "torque"):
        n, E, gn, ge, gk, gh = _gradient64(case, state)
        if kind == "energy":
            return {"E": E, "dn": gn.reshape(-1, 3), "deps": ge, "dK": gk, "dh": gh}
        return {"torque": _tangent(n, gn).reshape(-1, 3), "E": float(E), "dE_deps": float(ge),
                "dE_dK": float(gk), "dE_dh": float(gh)}
    if kind == "quench":
        return _quench64(case, state)
    if kind == "measure":
        return {"row": _row64(case, state)}
    if kind == "shells":
        return _shells64(case, state)
    return _stripes64(case, state)
