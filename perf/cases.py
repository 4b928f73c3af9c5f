"""The workloads this framework's speed is measured on.

Each case is work that a program using the TreePM engine has it do through
its public Python entry points (lageunha_b200.engine): force evaluations of
one box from 32^3 to 512^3 particles with both force laws, plain and from a
captured graph; the long-range part alone with the power spectrum on an odd
mesh; the drop-in entry points on host records; a global step of the
integrator; an ensemble of uneven boxes; served requests; groups; initial
conditions. The particle sets are the Zel'dovich-displaced lattices of
lageunha_b200/ic.py, with or without Plummer spheres, generated here with
torch on the GPU from the seed alone.

exact() restates each path in 64 bits with torch: the mesh force by plain FFTs,
the short-range force by a direct sum over all pairs inside the cut.
"""
import math
import random
import types

import numpy as np
import torch

from lageunha_b200 import engine as E

EPS = 0.05  # Plummer softening, cells (1/20 of the mean spacing at one particle per cell)
LAWS = {
    # the benchmark's law: Gaussian split, interlaced grids
    "headline": {"law": "gaussian", "rs_split": 0.7, "rsphere": 3.5, "theta": 0.4, "efold": 0.9},
    # the ensemble's and the request loop's
    "box": {"law": "gaussian", "rs_split": 0.8, "rsphere": 4.0, "theta": 0.3, "efold": 0.9},
    # the reference's defaults
    "reference": {"law": "reference", "rs_split": 1.25, "rsphere": 4.0, "theta": 0.3, "efold": 0.9},
}
# fields: spectral index, damping (cells), rms displacement (lattice spacings)
FIELDS = {"plain": (-2.0, 0.5, 0.3), "box": (-2.0, 0.5, 1.0), "clustered": (-2.0, 0.5, 1.5), "strong": (-2.5, 0.5, 2.0)}
ASTEP = 0.1  # of an expansion factor of 4
COSMO = (0.26, 0.74, -1.0, 0.0, 48.0)  # omep, omeplam, wlam0, wlam1, amax
DEV = "cuda:0"


def listed():
    return [
        # a small box of a parameter study, evaluated again and again from its
        # captured graph: launches and latency
        {"name": "graph_32", "kind": "forces", "mesh": 32, "np": 32768, "field": "box", "law": "box", "parts": 3, "graph": True},
        # the reference's default law on its smallest published set-up
        {"name": "plain_64", "kind": "forces", "mesh": 64, "np": 262144, "field": "plain", "law": "reference", "parts": 3, "graph": False},
        # long-range force and power spectrum of a ragged particle set on an odd mesh
        {"name": "spectrum_135", "kind": "spectrum", "mesh": 135, "np": 2000003, "field": "strong"},
        # the drop-in calls on the caller's host records: pmmain, then TreeMain
        {"name": "dropin_96", "kind": "dropin", "mesh": 96, "np": 884736, "field": "clustered", "step": 30},
        # one synchronisation step of the integrator (PULL, PUSH, drift)
        {"name": "step_128", "kind": "step", "mesh": 128, "np": 2097152, "field": "strong", "law": "box", "sync": True},
        # an uneven ensemble in one graph launch
        {"name": "ensemble_16", "kind": "ensemble", "boxes": 16, "lo": 32, "hi": 100, "mix": 4, "law": "box"},
        # continuous batching: requests of different sizes and step counts
        {"name": "served_8", "kind": "served", "requests": 8, "lo": 32, "hi": 80, "steps": 4, "mix": 5, "law": "box"},
        # a clustered box: deep trees, dense tiles
        {"name": "clustered_256", "kind": "forces", "mesh": 256, "np": 16777216, "field": "clustered", "law": "headline", "parts": 3, "graph": False},
        # the benchmark's headline, the largest box
        {"name": "scale_512", "kind": "forces", "mesh": 512, "np": 134217728, "field": "strong", "law": "headline", "parts": 3, "graph": False},
        # friends-of-friends groups of a clustered box
        {"name": "groups_160", "kind": "groups", "mesh": 160, "np": 4096000, "field": "clustered", "link": 0.2, "members": 20},
        # first-order initial conditions of a middle-sized run
        {"name": "zeldovich_256", "kind": "ic", "mesh": 256, "order": 1, "fnl": 0.0},
        # second-order ones with local non-Gaussianity
        {"name": "lpt2_120", "kind": "ic", "mesh": 120, "order": 2, "fnl": 50.0},
    ]


def _smooth(lo, hi):
    """The mesh sizes 2^a 3^b 5^c in [lo, hi]."""
    out = []
    for m in range(lo, hi + 1):
        k = m
        for p in (2, 3, 5):
            while k % p == 0:
                k //= p
        if k == 1:
            out.append(m)
    return out


def _log_mesh(rng, lo, hi):
    t = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(_smooth(lo, hi), key=lambda m: abs(math.log(m / t)))


def draw(rng):
    kind = rng.choice(["forces", "forces", "forces", "forces", "spectrum", "dropin", "step", "ensemble", "served", "groups", "ic"])
    if kind == "ensemble":
        lo = rng.randint(20, 48)
        return {"kind": kind, "boxes": rng.randint(3, 20), "lo": lo, "hi": rng.randint(lo + 8, 110), "mix": rng.randrange(1 << 30), "law": rng.choice(["box", "headline", "reference"])}
    if kind == "served":
        lo = rng.randint(20, 40)
        return {"kind": kind, "requests": rng.randint(2, 10), "lo": lo, "hi": rng.randint(lo + 8, 90), "steps": rng.randint(1, 4), "mix": rng.randrange(1 << 30), "law": rng.choice(["box", "headline"])}
    lo, hi = {"forces": (16, 320), "spectrum": (16, 320), "dropin": (24, 128), "step": (24, 256), "groups": (24, 200), "ic": (24, 320)}[kind]
    n = _log_mesh(rng, lo, hi)
    if kind == "ic":
        return {"kind": kind, "mesh": n, "order": rng.choice([1, 2]) if n <= 200 else 1, "fnl": rng.choice([0.0, 50.0])}
    # particle counts around one per cell, ragged ones among them
    np_ = n ** 3 if rng.random() < 0.4 else max(1000, int(n ** 3 * math.exp(rng.uniform(-0.7, 0.3))))
    c = {"kind": kind, "mesh": n, "np": np_, "field": rng.choice(["plain", "box", "clustered", "strong"])}
    if kind == "forces":
        c.update(law=rng.choice(["headline", "box", "reference"]), parts=rng.choice([3, 3, 3, 2, 1]), graph=rng.random() < 0.3)
    elif kind == "dropin":
        c.update(step=rng.choice([5, 15, 30, 100]))
    elif kind == "step":
        c.update(law=rng.choice(["headline", "box", "reference"]), sync=rng.random() < 0.5)
    elif kind == "groups":
        c.update(field="clustered", link=round(rng.uniform(0.12, 0.25), 3), members=rng.choice([5, 20, 32]))
    return c


# ------------------------------------------------------------------ inputs
def _displacement(n, seed, index, damp, rms):
    """Zel'dovich displacement (3 fields, lattice spacings) of a Gaussian field with P(k) ~ k^index exp(-(damp k)^2)."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    wk = torch.fft.rfftn(torch.randn((n, n, n), generator=g, device=DEV))
    f = torch.fft.fftfreq(n, device=DEV) * (2 * math.pi)
    fr = torch.fft.rfftfreq(n, device=DEV) * (2 * math.pi)
    ks = (fr[None, None, :], f[None, :, None], f[:, None, None])
    k2 = ks[0] ** 2 + ks[1] ** 2 + ks[2] ** 2
    k2[0, 0, 0] = 1.0
    wk *= torch.pow(k2, index / 4.0) * torch.exp(-0.5 * damp * damp * k2) / k2
    wk[0, 0, 0] = 0
    del k2
    psi = [torch.fft.irfftn(1j * k * wk, s=(n, n, n)) for k in ks]
    scale = rms / math.sqrt(sum(float((p.double() ** 2).mean()) for p in psi))
    return [p * scale for p in psi]


def _fixed(x, n):
    """uint32 fixed point (as int32) of positions in cells."""
    u = torch.remainder(torch.round(torch.remainder(x / n, 1.0) * 4294967296.0), 4294967296.0).to(torch.int64)
    return torch.where(u >= 2 ** 31, u - 2 ** 32, u).to(torch.int32)


def _particles(n, np_, field, seed, vel=False):
    """(np_, 3) fixed-point positions of a displaced lattice on an n^3 mesh, and velocities along
    psi, their rms 0.5 / n: a step of ASTEP then drifts 0.05 cells, and its kick is no small change."""
    index, damp, rms = FIELDS[field]
    m = max(2, round(np_ ** (1.0 / 3.0)))
    while m ** 3 < np_:
        m += 1
    psi = _displacement(m, seed, index, damp, rms)
    keep = None
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) + 17)
    if m ** 3 > np_:  # a ragged count: random lattice points left out
        keep = torch.randperm(m ** 3, generator=g, device=DEV)[:np_].sort().values
    pos = torch.empty((np_, 3), dtype=torch.int32, device=DEV)
    v = torch.empty((np_, 3), dtype=torch.float32, device=DEV) if vel else None
    sphere = None
    if field == "clustered":  # Plummer spheres in place of random field particles
        rng = np.random.Generator(np.random.PCG64(int(seed) + 7919))
        lo, hi = (2000, 20000) if n >= 128 else (200, 2000)
        cnt = rng.integers(lo, hi + 1, size=max(1, round(200 * (n / 256.0) ** 3)))
        cnt = cnt[np.cumsum(cnt) <= np_ // 3]
        total = int(cnt.sum())
        where = torch.randperm(np_, generator=g, device=DEV)[:total]
        centre = torch.from_numpy(rng.random((len(cnt), 3)) * n).to(DEV)
        r = 0.64 / torch.sqrt((torch.rand(total, generator=g, device=DEV, dtype=torch.float64) * 0.99) ** (-2.0 / 3.0) - 1.0)
        d = torch.randn((total, 3), generator=g, device=DEV, dtype=torch.float64)
        sphere = centre[torch.from_numpy(np.repeat(np.arange(len(cnt)), cnt)).to(DEV)] + d / d.norm(dim=1, keepdim=True) * r[:, None]
    q = torch.arange(m, device=DEV, dtype=torch.float64)
    for a in range(3):
        shape = [1, 1, 1]
        shape[2 - a] = m
        x = (psi[a].double() + q.view(shape)).reshape(-1)
        x = (x if keep is None else x[keep]) * (n / m)
        if sphere is not None:
            x[where] = sphere[:, a]
        pos[:, a] = _fixed(x, n)
        if vel:
            w = psi[a].reshape(-1)
            v[:, a] = (w if keep is None else w[keep]) * (0.5 / n / rms)
            if sphere is not None:
                v[where, a] = 0.0
    return pos, v


def _mix(case, count):
    """(lattice, mesh, steps) of the boxes of an ensemble or of the requests of a mix: log-uniform lattice sizes."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(count):
        m = round(math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]))))
        out.append((m, min(_smooth(12, 400), key=lambda k: abs(k - m)), r.randint(1, case.get("steps", 1))))
    return out


def _records(pos, vel, n, dtype):
    """Host records in the reference's layout: lattice index and float offset."""
    x = (pos.to(torch.int64) & 0xFFFFFFFF).double() * (n / 4294967296.0)
    cell = torch.floor(x).clamp(0, n - 1)
    r = np.zeros(pos.shape[0], dtype)
    ci = cell.to(torch.int64)
    r["indx"] = (ci[:, 0] + n * (ci[:, 1] + n * ci[:, 2])).cpu().numpy().astype(np.uint64)
    off, v = (x - cell).float().cpu().numpy(), vel.cpu().numpy()
    for a, k in enumerate("xyz"):
        r[k] = off[:, a]
        r["v" + k] = v[:, a]
    return r


def _velpot(n):
    """A smooth amplitude table over integer k^2, the rms displacement about a cell."""
    k2 = np.arange((n // 2) ** 2 + 1, dtype=np.float64)
    rk = np.sqrt(np.maximum(k2, 1.0))
    v = 0.05 * n ** 2 * rk ** -2.5 / (1.0 + (rk / (0.25 * n)) ** 2)
    v[0] = 0.0
    return v.astype(np.float32)


def _ic_seed(seed):
    return -(1 + int(seed) % 1000003)


def _ic_args(case):
    n = case["mesh"]
    if case["order"] == 1:
        return {"fnl": case["fnl"], "vamp": 0.01, "pfact": float(n)}
    return {"fnl": case["fnl"], "vamp": 0.01, "vamp2": -0.004, "damp1": 1.0, "damp2": -3.0 / 7.0, "pfact": 1.0 / n,
            "boxsize": 100.0, "omep": 0.26, "amax": 48.0, "growth": 0.02}


def prepare(case, seed):
    kind = case["kind"]
    s = types.SimpleNamespace(kind=kind, case=case)
    if kind in ("forces", "spectrum", "step", "groups"):
        n = case["mesh"]
        s.pos, s.vel = _particles(n, case["np"], case["field"], seed, vel=kind == "step")
        s.eng = E.Engine(n, epsilon=EPS, **LAWS[case.get("law", "reference")])
        s.out = torch.empty((case["np"], 3), dtype=torch.float32, device=DEV)
        if kind == "spectrum":
            s.eng.measure_power_spectrum(True)
        if kind == "step":
            s.cosmo = E.cosmology(*COSMO)
            s.new = torch.empty_like(s.pos)
            s.stream = torch.cuda.ExternalStream(s.eng.stream)
    elif kind == "dropin":
        n = case["mesh"]
        pos, _ = _particles(n, case["np"], case["field"], seed)
        vel = torch.zeros((case["np"], 3))
        s.dm, s.tdm = [(r.copy(), r) for r in (_records(pos, vel, n, d) for d in (E.DM_DTYPE, E.TREEDM_DTYPE))]
        s.eng = E.Engine(n, epsilon=EPS, **LAWS["reference"])
    elif kind in ("ensemble", "served"):
        sizes = _mix(case, case["boxes" if kind == "ensemble" else "requests"])
        sets = [_particles(n, m ** 3, ["box", "strong", "plain"][i % 3], seed * 64 + i, vel=True) for i, (m, n, _) in enumerate(sizes)]
        if kind == "ensemble":
            s.pos = [p for p, _ in sets]
            s.eng = [E.Engine(n, epsilon=EPS, **LAWS[case["law"]]) for _, n, _ in sizes]
            s.batch = E.Batch(s.eng)
            s.out = [torch.empty(p.shape, dtype=torch.float32, device=DEV) for p in s.pos]
        else:
            s.cosmo, s.sizes = E.cosmology(*COSMO), sizes
            host = lambda t: t.cpu().pin_memory()  # noqa: E731
            s.pos = [host(p).numpy().view(np.uint32) for p, _ in sets]
            s.vel = [host(v).numpy() for _, v in sets]
            s.new = [host(torch.empty_like(p)).numpy().view(np.uint32) for p, _ in sets]
            s.out = [host(torch.empty_like(v)).numpy() for _, v in sets]
            s.srv = E.Server(hbm_cap_bytes=40 * 10 ** 9, max_active=16, reserve_bytes=4 << 30)
    elif kind == "ic":
        n = case["mesh"]
        s.velpot, s.seed, s.args = _velpot(n), _ic_seed(seed), _ic_args(case)
        s.out = torch.empty((n ** 3, 8), dtype=torch.float32, device=DEV)
    return s


def run(s):
    c = s.case
    if s.kind == "forces":
        s.eng.load_fixed(s.pos)
        (s.eng.graph_compute if c["graph"] else s.eng.compute)(c["parts"])
        return s.eng.forces(s.out)
    if s.kind == "spectrum":
        s.eng.load_fixed(s.pos)
        s.eng.compute(E.PART_PM)
        p = s.eng.power_spectrum(100.0)
        return {"force": s.eng.forces(s.out), "pk": p["pk"], "cor": p["cor"], "sigma8": p["sigma8"]}
    if s.kind == "dropin":
        (dm, dm0), (tdm, tdm0) = s.dm, s.tdm
        np.copyto(dm, dm0)  # the calls add to the records' velocities
        np.copyto(tdm, tdm0)
        s.eng.pmmain(dm, 0.7)
        s.eng.treemain(tdm, 0.7, c["step"])
        return {"pm": [dm["vx"], dm["vy"], dm["vz"]], "tree": [tdm["vx"], tdm["vy"], tdm["vz"]]}
    if s.kind == "step":
        s.eng.load_fixed(s.pos, s.vel)
        s.eng.global_step(s.cosmo, 4.0, ASTEP, 30, sync=c["sync"])
        s.eng.velocities(s.out)
        s.eng.positions(s.new)
        with torch.cuda.stream(s.stream):  # the drift of every particle, cells
            moved = (s.new - s.pos).to(torch.float32) * (c["mesh"] / 4294967296.0)
        return {"vel": s.out, "moved": moved}
    if s.kind == "ensemble":
        for e, p in zip(s.eng, s.pos):
            e.load_fixed(p)
        s.batch.compute(E.PART_ALL)
        return [e.forces(o) for e, o in zip(s.eng, s.out)]
    if s.kind == "served":
        law = LAWS[c["law"]]
        for i, (_, n, steps) in enumerate(s.sizes):
            s.srv.submit(s.pos[i], s.vel[i], n_mesh=n, nsteps=steps, anow=4.0, astep=ASTEP, cosmo=s.cosmo, pos_out=s.new[i], vel_out=s.out[i], epsilon=EPS, **law)
        s.srv.wait(-1, 600.0)
        move = lambda a, b, n: (torch.from_numpy(b.view(np.int32)) - torch.from_numpy(a.view(np.int32))).float().mul_(n / 4294967296.0)  # noqa: E731
        return {"vel": list(s.out), "moved": [move(a, b, n) for a, b, (_, n, _) in zip(s.pos, s.new, s.sizes)]}
    if s.kind == "groups":
        s.eng.load_fixed(s.pos)
        labels, count = s.eng.fof(c["link"], c["members"])
        return {"labels": labels, "groups": count}
    if c["order"] == 1:
        E.ic_zeldovich(c["mesh"], s.seed, s.velpot, out=s.out, **s.args)
    else:
        E.ic_2lpt(c["mesh"], s.seed, s.velpot, out=s.out, **s.args)
    return {"indx": s.out.view(torch.int64)[:, 0], "field": s.out[:, 2:]}


# ------------------------------------------------------------------ what a pass needs
def _fft_flops(n, count):
    return count * 2.5 * n ** 3 * math.log2(n ** 3)


def _force_work(np_, n, law, parts):
    """Positions in, forces out; the transforms, and the pairs inside the cut of an unclustered set (20 flops each)."""
    L = LAWS[law]
    f = 0.0
    if parts & 1:
        f += _fft_flops(n, 4 if L["law"] == "gaussian" else 2) + np_ * 2 * 27 * 8
    if parts & 2:
        f += np_ * (np_ / n ** 3) * 4.18879 * L["rsphere"] ** 3 * 20
    return {"bytes": 24.0 * np_, "flops": f}


def work(case):
    k = case["kind"]
    if k == "forces":
        return _force_work(case["np"], case["mesh"], case["law"], case["parts"])
    if k == "spectrum":
        return _force_work(case["np"], case["mesh"], "reference", 1)
    if k == "dropin":
        a = _force_work(case["np"], case["mesh"], "reference", 3)
        return {"bytes": 2.0 * (32 + 40) * case["np"], "flops": a["flops"]}
    if k == "step":
        a = _force_work(case["np"], case["mesh"], case["law"], 3)
        return {"bytes": 48.0 * case["np"], "flops": a["flops"]}
    if k in ("ensemble", "served"):
        tot = {"bytes": 0.0, "flops": 0.0}
        for m, n, steps in _mix(case, case["boxes" if k == "ensemble" else "requests"]):
            a = _force_work(m ** 3, n, case["law"], 3)
            tot["bytes"] += 24.0 * m ** 3 * (1 if k == "ensemble" else 2)
            tot["flops"] += a["flops"] * (1 if k == "ensemble" else steps)
        return tot
    if k == "groups":
        return {"bytes": 16.0 * case["np"], "flops": case["np"] * 8.0 * (1 + 4.18879 * case["link"] ** 3)}
    n = case["mesh"]
    return {"bytes": 32.0 * n ** 3, "flops": _fft_flops(n, 5 if case["order"] == 1 else 14) + 60.0 * n ** 3}


def tolerance(case):
    """About four times what each path is off its 64-bit restatement."""
    k = case["kind"]
    if k == "groups":
        return "exact"  # the partition is unique, labels are whole numbers
    if k == "ic":
        return {"rel": 4e-5, "max": 2e-3}  # 32-bit transforms of a steep spectrum
    if k == "spectrum" or (k == "forces" and case["parts"] == 1):
        return {"rel": 2e-5, "max": 1e-3}  # 32-bit sums and transforms
    if k in ("step", "served"):
        return {"rel": 1.5e-4, "max": 0.01}  # a kick's share of the velocity, times the forces' error
    # tree forces: two correct walks accept other nodes under the same opening
    # angle, worst where the force nearly cancels (a barely displaced lattice)
    return {"rel": 1e-3, "max": 0.05}


# ------------------------------------------------------------------ 64-bit restatements
PM_FIT = (1.0 / 65536.0, 0.78224, 0.37971e-6, -0.60338, -0.34419e-7, -3.9741, -1.0607, -0.38145)


def _cells(pos, n):
    return (pos.to(torch.int64) & 0xFFFFFFFF).double() * (n / 4294967296.0)


def _tsc(x, n, fn):
    """fn(flat node index, weight) for the 27 TSC nodes of every particle."""
    near = torch.floor(x + 0.5)
    d = x - near
    w = (0.5 * (0.5 - d) ** 2, 0.75 - d * d, 0.5 * (0.5 + d) ** 2)
    ni = near.to(torch.int64)
    for c in range(3):
        for b in range(3):
            for a in range(3):
                i = torch.remainder(ni[:, 0] + a - 1, n) + n * (torch.remainder(ni[:, 1] + b - 1, n) + n * torch.remainder(ni[:, 2] + c - 1, n))
                fn(i, w[a][:, 0] * w[b][:, 1] * w[c][:, 2])


def _deposit(x, n):
    rho = torch.zeros(n ** 3, dtype=torch.float64, device=x.device)
    _tsc(x, n, lambda i, w: rho.index_add_(0, i, w))
    return rho.view(n, n, n)


def _modes(n):
    f = torch.arange(n, device=DEV, dtype=torch.float64)
    f = torch.where(f > n / 2.0, f - n, f)
    fx = torch.arange(n // 2 + 1, device=DEV, dtype=torch.float64)
    return fx[None, None, :], f[None, :, None], f[:, None, None]


def _interp(x, n, phi, coef):
    out = torch.zeros_like(x)
    for a in range(3):
        g = torch.zeros_like(phi)
        for j, c in enumerate(coef, 1):
            g += c * (torch.roll(phi, j, 2 - a) - torch.roll(phi, -j, 2 - a))
        g = g.reshape(-1)
        _tsc(x, n, lambda i, w: out[:, a].add_(w * g[i]))
    return out


def _pm_exact(x, n, law):
    """(long-range force, spectrum of the density)."""
    kx, ky, kz = _modes(n)
    k2 = kx ** 2 + ky ** 2 + kz ** 2
    k2[0, 0, 0] = 1.0
    back = lambda s: torch.fft.irfftn(s, s=(n, n, n), norm="forward")  # noqa: E731
    r1 = torch.fft.rfftn(_deposit(x, n))
    if law["law"] == "reference":
        g = -1.0 / math.pi / k2 * torch.exp(-k2 * (math.pi * np.float32(law["efold"]).item() / n) ** 2) / n ** 3
        g[0, 0, 0] = 0.0
        return _interp(x, n, back(r1 * g), (2.0 / 3.0, -1.0 / 12.0)), r1
    rs = np.float32(law["rs_split"]).item()
    coef = (4.0 / 5.0, -1.0 / 5.0, 4.0 / 105.0, -1.0 / 280.0)
    ks = [2 * math.pi / n * k for k in (kx, ky, kz)]
    D = [sum(2 * c * torch.sin((j + 1) * k) for j, c in enumerate(coef)) for k in ks]
    D2 = D[0] ** 2 + D[1] ** 2 + D[2] ** 2
    num, den = torch.zeros_like(k2), torch.zeros_like(k2)
    for ax in range(-2, 3):
        for ay in range(-2, 3):
            for az in range(-2, 3):
                if (ax + ay + az) & 1:
                    continue
                q = [k + 2 * math.pi * m for k, m in zip(ks, (ax, ay, az))]
                u = 1.0
                for v in q:
                    u = u * torch.special.sinc(v / (2 * math.pi)) ** 6
                q2 = q[0] ** 2 + q[1] ** 2 + q[2] ** 2
                R = -1.0 / math.pi / (q2 * (n / (2 * math.pi)) ** 2).clamp_min(1e-300) * torch.exp(-q2 * rs * rs)
                num += u * R * (D[0] * q[0] + D[1] * q[1] + D[2] * q[2])
                den += u
    ok = (D2 > 0) & (k2 + 0 * kx > 0)
    if n % 2 == 0:
        h = n / 2.0
        ok = ok & (kx.abs() != h) & (ky.abs() != h) & (kz.abs() != h)
    ok[0, 0, 0] = False
    g = torch.where(ok, num / (D2 * den * den).clamp_min(1e-300) / n ** 3, torch.zeros_like(num))
    th = math.pi / n * (kx + ky + kz)
    ph = torch.polar(torch.ones_like(th), th)
    r2 = torch.fft.rfftn(_deposit(x + 0.5, n))
    s = 0.5 * (r1 + ph * r2) * g
    return 0.5 * (_interp(x, n, back(s), coef) + _interp(x + 0.5, n, back(s * ph.conj()), coef)), r1


def _law(r2, law):
    """-(short-range force)/r of a unit mass."""
    r = torch.sqrt(r2).clamp_min(1e-9)
    soft = r / (r2 + np.float32(EPS).item() ** 2) ** 1.5
    if law["law"] == "reference":
        P = PM_FIT
        far = torch.tanh(P[1] * r) / r ** 2 - P[1] / (torch.cosh(P[1] * r) ** 2 * r) - 2 * P[2] / P[0] * r * torch.exp(P[3] * r ** 2) \
            - 2 * P[2] * P[3] / P[0] * r ** 3 * torch.exp(P[3] * r ** 2) + P[4] / P[0] * (1 + P[5] * r ** 2 + P[6] * r ** 4) * torch.exp(P[7] * r ** 2)
    else:
        u = r / (2 * np.float32(law["rs_split"]).item())
        far = (torch.special.erf(u) - 2 * u / math.sqrt(math.pi) * torch.exp(-u * u)) / r ** 2
    return -(soft - far) / r


def _tree_exact(x, n, law, pairs_most):
    """Direct short-range sum over every pair inside the cut; None if the cell lists hold more than pairs_most pairs."""
    rc = np.float32(law["rsphere"]).item()
    nc = int(n // rc)
    cell = torch.clamp((x * (nc / n)).to(torch.int64), max=nc - 1)
    cid = cell[:, 0] + nc * (cell[:, 1] + nc * cell[:, 2])
    order = torch.argsort(cid)
    xs, cs = x[order], cell[order]
    cnt = torch.bincount(cid, minlength=nc ** 3)
    start = torch.cumsum(cnt, 0) - cnt
    offs = [(a, b, c) for c in (-1, 0, 1) for b in (-1, 0, 1) for a in (-1, 0, 1)] if nc >= 3 else \
        [(a, b, c) for c in range(nc) for b in range(nc) for a in range(nc)]
    out = torch.zeros_like(xs)
    nbr = []
    for o in offs:
        t = [torch.remainder(cs[:, a] + o[a], nc) for a in range(3)]
        nbr.append(t[0] + nc * (t[1] + nc * t[2]))
    total = sum(cnt[b] for b in nbr)
    if float(total.sum()) > pairs_most:
        return None
    cum = torch.cumsum(total, 0).cpu().numpy()
    i0, np_ = 0, x.shape[0]
    while i0 < np_:
        base = cum[i0 - 1] if i0 else 0
        i1 = max(i0 + 1, int(np.searchsorted(cum, base + (1 << 26), side="right")))
        for b in nbr:
            c = cnt[b[i0:i1]]
            m = int(c.sum())
            if not m:
                continue
            t = torch.repeat_interleave(torch.arange(i0, i1, device=x.device), c, output_size=m)
            first = torch.cumsum(c, 0) - c
            j = torch.arange(m, device=x.device) - torch.repeat_interleave(first - start[b[i0:i1]], c, output_size=m)
            d = xs[t] - xs[j]
            d -= n * torch.round(d / n)
            r2 = (d * d).sum(1)
            w = torch.where((r2 <= rc * rc) & (j != t), _law(r2, law), torch.zeros_like(r2))
            out.index_add_(0, t, d * w[:, None])
        i0 = i1
    f = torch.empty_like(out)
    f[order] = out / n ** 2
    return f


def _force_exact(pos, n, law, parts, pairs_most=9e10):
    x = _cells(pos, n)
    f = torch.zeros_like(x)
    if parts & 2:
        t = _tree_exact(x, n, law, pairs_most)
        if t is None:
            return None
        f += t
    if parts & 1:
        f += _pm_exact(x, n, law)[0]
    return f


def _hof(a):
    om, ol, _, _, am = COSMO
    z1 = am / a
    return math.sqrt(z1 ** 3 * om + z1 ** 2 * (1 - om - ol) + ol)


def _drag(a1, a2):
    return (a1 ** 3 * _hof(a1)) / (a2 ** 3 * _hof(a2))


def _kick(n, a1, a2):
    om, am = COSMO[0], COSMO[4]
    ap = lambda a: math.sqrt(8 * math.pi / 3 / (am * om) * (a / am) ** 2) * _hof(a)  # noqa: E731
    k = 200
    h = (a2 - a1) / k
    y = [1.0 / (a * ap(a)) for a in (a1 + h * i for i in range(k + 1))]
    s = h / 3 * (y[0] + y[-1] + 4 * sum(y[1:-1:2]) + 2 * sum(y[2:-1:2]))
    return s * n / (a2 * a2 * ap(a2))


def _step_exact(pos, vel, n, law, sync):
    x = _cells(pos, n)
    tree = _tree_exact(x, n, law, 9e10)
    if tree is None:
        return None
    pm = _pm_exact(x, n, law)[0]
    astep = np.float32(ASTEP).item()
    a, h = 4.0, 0.5 * astep
    full = _kick(n, a - h, a + h)
    v = vel.double()
    if sync:
        v = v * _drag(a - h, a) + _kick(n, a - h, a) * pm + full * tree
        v = v * _drag(a, a + h) + _kick(n, a, a + h) / _drag(a, a + h) * pm + full * tree
    else:
        v = v * _drag(a - h, a + h) + full * (pm + tree)
    return {"vel": v, "moved": v * (astep * n)}


def _spectrum_exact(r, n, boxsize):
    kx, ky, kz = _modes(n)
    k = torch.sqrt(kx ** 2 + ky ** 2 + kz ** 2)
    win = 1.0
    for m in (kx, ky, kz):
        win = win * torch.special.sinc(m / n) ** 3
    p = (r.abs() / n ** 3) ** 2 / win ** 2
    use = (2 * kx < n).expand_as(p)
    k, p = k[use], p[use]
    b = torch.floor(k).to(torch.int64)
    w = k - b
    s, ws = (torch.zeros(2 * n + 4, dtype=torch.float64, device=DEV) for _ in range(2))
    for bb, ww in ((b, 1 - w), (b + 1, w)):
        s.index_add_(0, bb, ww * p)
        ws.index_add_(0, bb, ww)
    s, ws = s[:n + 1].cpu().numpy(), ws[:n + 1].cpu().numpy()
    pk = np.where(ws > 0, s / np.maximum(ws, 1e-300), 0.0)
    pk[0] = s[0]
    i = np.arange(n + 1, dtype=np.float64)
    th = 2 * math.pi * 8.0 / boxsize * i[1:]
    sig = math.sqrt(4 * math.pi * 9.0 * float(np.sum(pk[1:] * i[1:] ** 2 * (np.sin(th) - th * np.cos(th)) ** 2 / th ** 6)))
    cor = np.zeros(n + 1)
    cor[1:] = 2 * n * (np.sin(2 * math.pi / n * np.outer(i[1:], i[1:])) @ (i[1:] * pk[1:])) / i[1:]
    return pk, cor, sig


def _gasdev(seed, count):
    """`count` accepted Box-Muller pairs (second deviate first) of Numerical Recipes' gasdev on ran3, in its 32-bit floats."""
    big = 1000000000
    ma = [0] * 56
    mj = (161803398 - abs(seed)) % big
    ma[55], mk = mj, 1
    for i in range(1, 55):
        ii = (21 * i) % 55
        ma[ii] = mk
        mk = (mj - mk) % big
        mj = ma[ii]
    for _ in range(4):
        for i in range(1, 56):
            ma[i] = (ma[i] - ma[1 + (i + 30) % 55]) % big
    trials = int(count * 4 / math.pi * 1.03) + 4096
    x = np.zeros(55 + 2 * trials + 24, np.int64)
    x[:55] = ma[1:]
    for t in range(55, 55 + 2 * trials, 24):  # x_t = x_{t-55} - x_{t-24}
        d = x[t - 55:t - 31] - x[t - 24:t]
        x[t:t + 24] = np.where(d < 0, d + big, d)
    u = (x[55:55 + 2 * trials] * 1e-9).astype(np.float32)
    v = (2.0 * u.astype(np.float64) - 1.0).astype(np.float32).reshape(-1, 2)
    r = v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1]
    ok = (r < 1.0) & (r > 0.0)
    v, r = v[ok][:count], r[ok][:count].astype(np.float64)
    fac = np.sqrt(-2.0 * np.log(r) / r)
    return np.stack([v[:, 1] * fac, v[:, 0] * fac], 1)


def _noise_exact(n, seed, velpot):
    kx, ky, kz = (m.to(torch.int64) for m in _modes(n))
    k2 = (kx ** 2 + ky ** 2 + kz ** 2).cpu().numpy()
    use = (k2 > 0) & (k2 <= (n // 2) ** 2)
    g = _gasdev(seed, int(use.sum()))
    spec = np.zeros(k2.shape, np.complex128)
    spec[use] = (g[:, 0] + 1j * g[:, 1]) * velpot.astype(np.float64)[k2[use]]
    p = spec[:, :, 0].copy()  # [z][y]: the reference's conjugate completion of kx = 0
    for k in range(1, n // 2):
        for j in range(n):
            if j != n // 2:
                spec[n - k, (n - j) % n, 0] = np.conj(p[k, j])
    for j in range(1, n // 2):
        spec[0, n - j, 0] = np.conj(p[0, j])
    return torch.from_numpy(spec).to(DEV)


def _ic_exact(case, seed):
    n, a = case["mesh"], _ic_args(case)
    kx, ky, kz = _modes(n)
    two_pi = float(np.float32(2 * math.pi))
    back = lambda s: torch.fft.irfftn(s, s=(n, n, n))  # noqa: E731
    s1 = _noise_exact(n, _ic_seed(seed), _velpot(n))
    f64 = lambda v: float(np.float32(v))  # noqa: E731
    if case["order"] == 1:
        phi = back(s1)
        var = (phi ** 2).mean() - phi.mean() ** 2
        s1 = torch.fft.rfftn(phi + f64(a["fnl"]) * (phi ** 2 - var))
        out = torch.empty((n ** 3, 6), dtype=torch.float64, device=DEV)
        below = (kx < n // 2).double()
        for i, k in enumerate((kx, ky, kz)):
            v = f64(a["vamp"]) ** 2 * back(1j * two_pi * k * below * s1).reshape(-1)
            out[:, i], out[:, 3 + i] = f64(a["pfact"]) * v, v
    else:
        if a["fnl"]:
            vp = 1.5 * (100.0 * a["boxsize"] / 2.99792458e5) ** 2 * f64(a["omep"]) * a["amax"]
            # the kx = n/2 element of an even padded row (the imaginary part of
            # an odd row's last element) is left unscaled both ways
            fr, fi = (torch.full((n // 2 + 1,), vp, dtype=torch.float64, device=DEV) for _ in range(2))
            fi[-1] = 1.0
            if n % 2 == 0:
                fr[-1] = 1.0
            s1 = torch.complex(s1.real * fr, s1.imag * fi)
            phi = back(s1)
            var = (phi ** 2).mean() - phi.mean() ** 2
            fz = 1.0 / f64(a["growth"]) / a["amax"]
            s1 = torch.fft.rfftn(phi + fz * a["fnl"] * (phi ** 2 - var))
            s1 = torch.complex(s1.real / fr, s1.imag / fi)
        h = lambda u, v: back(-two_pi ** 2 * u * v * s1)  # noqa: E731
        xx, yy, zz = h(kx, kx), h(ky, ky), h(kz, kz)
        src = xx * yy + xx * zz + yy * zz - h(ky, kx) ** 2 - h(kz, kx) ** 2 - h(kz, ky) ** 2
        k2 = kx ** 2 + ky ** 2 + kz ** 2
        k2[0, 0, 0] = 1.0
        s2 = torch.fft.rfftn(src) / (-k2 * two_pi ** 2)
        s2[0, 0, 0] = 0.0
        out = torch.empty((n ** 3, 6), dtype=torch.float64, device=DEV)
        for col, (b1, b2) in ((3, (a["vamp"], a["vamp2"])), (0, (a["pfact"] * a["damp1"], a["pfact"] * a["damp2"]))):
            for i, k in enumerate((kx, ky, kz)):
                out[:, col + i] = back(1j * two_pi * k * (f64(b1) * s1 + f64(b2) * s2)).reshape(-1)
    return {"indx": None, "field": out}


def exact(case, seed):
    kind = case["kind"]
    if kind == "groups":
        return None
    if kind == "ic":
        return _ic_exact(case, seed) if case["mesh"] <= 260 else None
    if kind in ("ensemble", "served"):
        sizes = _mix(case, case["boxes" if kind == "ensemble" else "requests"])
        vel, moved = [], []
        for i, (m, n, steps) in enumerate(sizes):
            pos, v = _particles(n, m ** 3, ["box", "strong", "plain"][i % 3], seed * 64 + i, vel=True)
            if kind == "ensemble":
                vel.append(_force_exact(pos, n, LAWS[case["law"]], 3))
            else:  # the first step's end is the start of the next: one-step requests only
                r = _step_exact(pos, v, n, LAWS[case["law"]], False) if steps == 1 else None
                vel.append(r and r["vel"])
                moved.append(r and r["moved"])
        return vel if kind == "ensemble" else {"vel": vel, "moved": moved}
    n, np_ = case["mesh"], case["np"]
    if np_ > 2e7:
        return None
    pos, v = _particles(n, np_, case["field"], seed, vel=kind == "step")
    if kind == "forces":
        return _force_exact(pos, n, LAWS[case["law"]], case["parts"])
    if kind == "spectrum":
        f, r = _pm_exact(_cells(pos, n), n, LAWS["reference"])
        pk, cor, sig = _spectrum_exact(r, n, 100.0)
        return {"force": f, "pk": pk, "cor": cor, "sigma8": sig}
    if kind == "step":
        return _step_exact(pos, v, n, LAWS[case["law"]], case["sync"])
    # the records' 32-bit offsets are what the engine is given
    r = _records(pos, torch.zeros((np_, 3)), n, E.DM_DTYPE)
    idx = torch.from_numpy(r["indx"].astype(np.int64)).to(DEV)
    grid = torch.stack([idx % n, idx // n % n, idx // (n * n)], 1).double()
    x = torch.remainder(grid + torch.from_numpy(np.stack([r["x"], r["y"], r["z"]], 1)).to(DEV).double(), float(n))
    tree = _tree_exact(x, n, LAWS["reference"], 9e10)
    fact = np.float32(0.7).item()
    pm = fact * _pm_exact(x, n, LAWS["reference"])[0]
    if tree is None:
        return {"pm": [pm[:, a] for a in range(3)], "tree": [None] * 3}
    tree = fact * tree
    return {"pm": [pm[:, a] for a in range(3)], "tree": [tree[:, a] for a in range(3)]}
