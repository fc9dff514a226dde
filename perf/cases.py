"""Workloads that the framework's speed is measured on, through its public entry points.

Every case is a plain dict; ``prepare`` makes what a program holds before the
call from a seed, ``run`` makes one pass, ``work`` says what a pass cannot do
without and ``exact`` gives the same outputs in 64 bits from plain torch.

Kinds of case
  march    the native step driver, ``Simulation``: either `steps` further
           steps of a run in progress, or (reload) a new initial state uploaded
           from pinned host memory and `steps` steps from it, as a sweep over
           scenarios does
  dropin   the reference's own step loop through the drop-in calls
           (``ReferenceStep``): search and re-sort before each stage, Adami,
           interaction, predictor, corrector
  search   one neighbour search over particles that moved since they were last
           sorted (``Grid.neighbor_search``, or the call that allocates nothing)
  pairs    one ``particle_interaction`` in a sorted state: in a grid of the
           caller's own (fresh lists), or in a grid of the library's
  wall     one ``adami_boundary``
  smooth   one ``stress_regularization``

The states are those of a flow under way: particles off their lattice by a few
percent of the spacing, a shear flow of a few per mille of the sound speed with
noise on it, geostatic stress with a few percent of noise.  Whole runs return
their arrays in the particles' original order (idep.w carries it), which no
search changes.
"""
import math

import numpy as np
import torch

import loquat_b200 as lq
from loquat_b200 import cases
from loquat_b200.dropin import ReferenceStep


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest scenario of the ensemble workload (5 k soil particles): launches and latency
        dict(name="column_5k_plain", kind="march", scene="column", nx=20, ny=10, nz=25, dr=0.002, hdr=1.2, mixed=False,
             steps=30, reload=True, wide=False, artp=False),
        # the column collapse of the reference's example, 50 k soil and 116 k wall particles
        dict(name="column_50k_mixed", kind="march", scene="column", nx=100, ny=10, nz=50, dr=0.002, hdr=1.2,
             mixed=True, steps=30, reload=True, wide=False, artp=False),
        # the benchmark's default workload, 1.97 M soil particles, mixed precision, a run in progress
        dict(name="cylinder_2m_mixed", kind="march", scene="cylinder", dr=0.002949, hdr=1.3, mixed=True, steps=10,
             reload=False, wide=False, artp=False),
        # the same geometry at an ordinary size in plain FP32 with the artificial stress on
        dict(name="cylinder_230k_plain", kind="march", scene="cylinder", dr=0.00603, hdr=1.3, mixed=False, steps=10,
             reload=False, wide=False, artp=True),
        # the von Wolffersdorff slope at its stated size, 2.85 M soil particles
        dict(name="slope_2m9_mixed", kind="march", scene="slope", dr=0.005, hdr=1.2, mixed=True, steps=10,
             reload=False, wide=False, artp=False),
        # batched ensemble: own materials and grid frames, more wall than soil, two-level lists
        dict(name="ensemble_24_mixed", kind="march", scene="ensemble", scenarios=24, dr=0.002, hdr=1.2, mixed=True,
             steps=10, reload=False, wide=True, artp=False),
        # the reference's call sequence, as a caller of its headers makes it, 0.79 M soil particles
        dict(name="dropin_cylinder_790k", kind="dropin", scene="cylinder", dr=0.004, hdr=1.3, model=1, steps=5),
        # the same sequence on a few thousand particles with the four-parameter hypoplastic law
        dict(name="dropin_small_hypo", kind="dropin", scene="small", nx=17, ny=9, nz=13, dr=0.002, hdr=1.2, model=2,
             steps=5),
        # a neighbour search alone, 2.3 M particles in 2.1 M cells
        dict(name="search_2m", kind="search", scene="cylinder", dr=0.002949, hdr=1.3, fixed=False),
        # pair sums for a caller with a grid of its own, at a ragged size
        dict(name="pairs_own_grid_111k", kind="pairs", scene="small", nx=61, ny=37, nz=49, dr=0.002, hdr=1.2, model=1,
             carry=False, artp=False),
        # boundary extrapolation where walls outnumber the soil (the column's 116 k wall particles)
        dict(name="wall_column_116k", kind="wall", scene="column", nx=100, ny=10, nz=50, dr=0.002, hdr=1.2),
        # the stress filter over 400 k soil particles, then nothing else
        dict(name="smooth_cylinder_400k", kind="smooth", scene="cylinder", dr=0.005, hdr=1.3),
    ]


def _spread(rng, lo, hi):
    """A whole number spread evenly over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["march", "march", "march", "dropin", "search", "pairs", "wall", "smooth"])
    hdr = rng.choice([1.2, 1.3])
    nx, ny, nz = _spread(rng, 9, 140), _spread(rng, 5, 40), _spread(rng, 9, 110)
    cyl_dr = math.exp(rng.uniform(math.log(0.003), math.log(0.02)))
    box = dict(scene="small", nx=nx, ny=ny, nz=nz, dr=0.002, hdr=hdr)
    cyl = dict(scene="cylinder", dr=cyl_dr, hdr=1.3)
    if kind == "march":
        reload = rng.random() < 0.4
        scene = rng.choice(["column", "cylinder", "slope", "ensemble"])
        c = dict(kind=kind, scene=scene, hdr=hdr, mixed=rng.random() < 0.6, steps=30 if reload else 10,
                 reload=reload, wide=rng.random() < 0.3, artp=rng.random() < 0.2)
        if scene == "column":
            c.update(nx=nx, ny=ny, nz=nz, dr=0.002)
        elif scene == "cylinder":
            c.update(dr=max(cyl_dr, 0.005) if reload else cyl_dr, hdr=1.3)
        elif scene == "slope":
            c.update(dr=math.exp(rng.uniform(math.log(0.009 if reload else 0.0055), math.log(0.03))), hdr=1.2)
        else:
            c.update(scenarios=_spread(rng, 2, 5 if reload else 22), dr=0.002, hdr=1.2)
        return c
    if kind == "dropin":
        return dict(rng.choice([box, cyl]), kind=kind, model=1, steps=rng.randint(2, 6))
    if kind == "search":
        return dict(rng.choice([box, cyl]), kind=kind, fixed=rng.random() < 0.3 and cyl_dr > 0.006)
    if kind == "pairs":
        return dict(rng.choice([box, cyl]), kind=kind, model=1, carry=rng.random() < 0.5, artp=rng.random() < 0.2)
    return dict(rng.choice([box, cyl]), kind=kind)


# ------------------------------------------------------------------- states
def _scene(case, seed):
    """The case's particle set with a flow under way, ids in idep.w."""
    scene, dr, hdr = case["scene"], case["dr"], case["hdr"]
    kw = dict(dr=dr, hdr=hdr, jitter_frac=0.05)
    if scene == "column":
        c = cases.column_collapse(length=case["nx"] * dr, thickness=case["ny"] * dr, height=case["nz"] * dr,
                                  runout=3 * case["nx"] * dr, seed=seed, **kw)
    elif scene == "cylinder":
        c = cases.cylinder_collapse(seed=seed, **kw)
    elif scene == "slope":
        c = cases.slope_failure(seed=seed, **kw)
    elif scene == "ensemble":
        # the workload's own scenarios, the same for every seed; their jitter is ours
        c = cases.ensemble(n=case["scenarios"], **dict(kw, jitter_frac=0.0))[0]
        jitter = np.random.default_rng([seed, 5]).uniform(-0.05 * dr, 0.05 * dr, (c.par.np, 3))
        c.pospres[:, :3] += jitter.astype(np.float32)
    else:
        c = cases.small_column(nsx=case["nx"], nsy=case["ny"], nsz=case["nz"], model=case.get("model", 1), seed=seed,
                               **kw)
    par = c.par
    if case.get("artp"):
        par.artificial_pressure, par.artificial_pressure_coefficient = 1, 0.3
        lq.initialize_parameters(par)
    rng = np.random.default_rng([seed, 17])
    nb, nm = par.npb, par.npm
    U = np.float32(0.004 * par.cs)
    z = c.pospres[nb:, 2] / c.pospres[nb:, 2].max()
    v = rng.random((nm, 3), dtype=np.float32)
    v -= 0.5
    v *= 0.2 * U
    v[:, 0] += U * z
    v[:, 2] -= 0.3 * U * z
    c.velrhop[nb:, :3] = v
    noise = rng.standard_normal((nm, 6), dtype=np.float32)
    noise *= 0.02 * np.abs(c.str_[nb:, 2:3])
    c.str_[nb:] += noise
    c.pospres[nb:, 3] = -(c.str_[nb:, 0] + c.str_[nb:, 1] + c.str_[nb:, 2]) / 3.0
    c.velrhop[nb:, 3] *= 1.0 + 1.0e-3 * (rng.random(nm, dtype=np.float32) - 0.5)
    c.idep[:, 3] = np.arange(par.np, dtype=np.float32)
    return c


class _Array:
    """A device array of the library, for torch.as_tensor; the tensor keeps the array's owner alive."""

    def __init__(self, ptr, shape, kind, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=kind, version=3)


def _view(owner, ptr, shape, kind="<f4"):
    return torch.as_tensor(_Array(ptr, shape, kind, owner), device="cuda")


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _par_device(par):
    return torch.from_numpy(np.frombuffer(par.to_bytes(), np.uint8).copy()).cuda()


def _order(c):
    """The sorted order of the particles in the reference's grid and its cell bounds."""
    par = c.par
    par.dt = par.cfl * par.h / par.cs
    g, pd, pos = lq.Grid(par.np, par.ncell), _par_device(par), _device(c.pospres)
    g.neighbor_search(par, pd, pos)
    a = g.arrays()
    idx = _view(g, a["part_idx"], (par.np,), "<i4").long()
    beg = _view(g, a["cell_beg"], (par.ncell,), "<i4").clone()
    end = _view(g, a["cell_end"], (par.ncell,), "<i4").clone()
    torch.cuda.synchronize()
    return g, pd, idx, beg, end


def _sorted(case, seed):
    """A sorted state on the device, as a caller holds it between search and stage."""
    c = _scene(case, seed)
    g, pd, idx, beg, end = _order(c)
    arrays = [_device(a)[idx].contiguous() for a in c.arrays()]
    torch.cuda.synchronize()
    return c.par, pd, g, beg, end, arrays


def _slot_sorted(case, seed):
    """The same order from plain torch, with the arrays in 64 bits (the oracle's inputs)."""
    c = _scene(case, seed)
    idx = torch.sort(_keys(c.par, torch.from_numpy(c.pospres)), stable=True)[1]
    c.par.dt = c.par.cfl * c.par.h / c.par.cs
    return c.par, [torch.from_numpy(np.ascontiguousarray(a))[idx].to(_DEV()).double() for a in c.arrays()]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "march":
        c = _scene(case, seed)
        sim = lq.Simulation(c.par, *c.arrays(), graph=True, mixed=case["mixed"])
        if "materials" in c.meta:
            sim.set_materials(c.meta["materials"])
            sim.set_frames(c.meta["frames"])
        if "hypoplastic" in c.meta:
            sim.set_hypoplastic(c.meta["hypoplastic"])
        if case["wide"]:
            sim.set_skin(0.02)
            sim.set_wide_skin(0.22)
        host = [torch.from_numpy(np.ascontiguousarray(a)).pin_memory() for a in c.arrays()] if case["reload"] else None
        out = [torch.empty((c.par.np, w), device="cuda") for w in (4, 4, 2, 6, 6)]
        torch.cuda.synchronize()
        return dict(case=case, sim=sim, host=host, out=out, stream=torch.cuda.ExternalStream(sim.stream()))
    if kind == "dropin":
        c = _scene(case, seed)
        r = ReferenceStep(c.par, *c.arrays())
        return dict(case=case, step=r, out=[torch.empty((c.par.np, w), device="cuda") for w in (4, 4, 2, 6, 6)])
    if kind == "search":
        # sorted once, then moved by up to a tenth of the smoothing length: a few percent change their cell
        c = _scene(case, seed)
        g, pd, idx, beg, end = _order(c)
        pos = _device(c.pospres)[idx].contiguous()
        gen = torch.Generator(device="cuda").manual_seed(seed)
        pos[:, :3] += (torch.rand(pos.shape[0], 3, device="cuda", generator=gen) - 0.5) * (0.2 * c.par.h)
        n, ncell = c.par.np, c.par.ncell
        a = g.arrays()
        out = [_view(g, a["part_cel"], (n,), "<i4"), _view(g, a["part_idx"], (n,), "<i4"),
               _view(g, a["cell_beg"], (ncell,), "<i4"), _view(g, a["cell_end"], (ncell,), "<i4")]
        if case["fixed"]:
            out = [torch.empty_like(t) for t in out]
        return dict(case=case, par=c.par, pd=pd, grid=g, pos=pos, out=out)
    par, pd, g, beg, end, arrays = _sorted(case, seed)
    s = dict(case=case, par=par, pd=pd, grid=g, beg=beg, end=end, state=arrays)
    n = par.np
    if kind == "pairs":
        if case["carry"]:
            a = g.arrays()
            s["beg"], s["end"] = a["cell_beg"], a["cell_end"]
        lq.interaction_reserve(par)
        s["rates"] = [torch.zeros(n, w, device="cuda") for w in (4, 4, 6)]
    elif kind == "smooth":
        s["cache"] = torch.zeros(n, 6, device="cuda")
    return s


# --------------------------------------------------------------------- runs
def _by_id(state, out):
    """The state arrays in the particles' original order; of idep the plastic strain and the void ratio
    (the object id and the order are the caller's own tags)."""
    at = state[2][:, 3].long()
    for a, o in zip((state[0], state[1], state[2][:, 1:3], state[3], state[4]), out):
        o.index_copy_(0, at, a)
    return dict(zip(("pos", "vel", "idep", "str", "stn"), out))


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "march":
        sim = s["sim"]
        if s["host"] is not None:
            sim.upload(*s["host"])
        sim.step(case["steps"])
        with torch.cuda.stream(s["stream"]):
            n, p = sim.np, sim.state_pointers()
            state = [_view(sim, p[k], (n, w)) for k, w in (("pospres", 4), ("velrhop", 4), ("idep", 4), ("str", 6),
                                                      ("stn", 6))]
            return _by_id(state, s["out"])
    if kind == "dropin":
        s["step"].step(case["steps"])
        return _by_id(s["step"].state, s["out"])
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "search":
        if case["fixed"]:
            lq.grid_neighbor_search_noalloc(s["par"], s["pd"], s["pos"], *s["out"], stream=stream)
        else:
            s["grid"].neighbor_search(s["par"], s["pd"], s["pos"], stream=stream)
        return s["out"]
    par, pd, st, nb = s["par"], s["pd"], s["state"], s["par"].npb
    if kind == "pairs":
        lq.particle_interaction(par, pd, *st, *s["rates"], s["beg"], s["end"], stream=stream)
        return [r[nb:] for r in s["rates"]]
    if kind == "wall":
        lq.adami_boundary(par, pd, st[0], st[1], st[3], s["beg"], s["end"], stream=stream)
        return st[3]
    lq.stress_regularization(par, pd, st[0], st[1], st[3], s["cache"], s["beg"], s["end"], stream=stream)
    return st[3]


# --------------------------------------------------------------------- work
def _counts(case):
    """Soil and wall particles and cells of a case, from its geometry."""
    scene, dr = case["scene"], case["dr"]
    h2 = 2.0 * case["hdr"] * dr
    if scene == "column":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        nw = round(1.1 * nz)
        walls = (3 * nx + 3) * (ny + 6) * 3 + 3 * ny * nw + 2 * (3 * nx + 3) * 3 * nw
        cells = 2 * ((3 * nx + 3) * dr / h2 + 1) * ((ny + 6) * dr / h2 + 1) * ((1.5 * nz + 3) * dr / h2 + 1)
        return nx * ny * nz, walls, cells
    if scene == "cylinder":
        return math.pi * 0.04 * 0.4 / dr ** 3, 3.0 / dr ** 2, 2 * (1.0 / h2 + 1) ** 2 * ((3 * dr + 0.46) / h2 + 1)
    if scene == "slope":
        walls = 3 * 3.0 * 0.35 / dr ** 2 + 2 * 3 * 3.0 * 0.66 / dr ** 2
        return (2.0 - 0.3) * 0.6 * 0.35 / dr ** 3, walls, 2 * 3.0 * 0.38 * 0.93 / h2 ** 3
    if scene == "ensemble":
        return 54000.0 * case["scenarios"], 63000.0 * case["scenarios"], 2.0e5 * case["scenarios"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    walls = (nx + 16) * (ny + 6) * 3 + 3 * ny * (nz + 2) + 2 * (nx + 16) * 3 * (nz + 2)
    return nx * ny * nz, walls, 2 * ((nx + 16) * dr / h2 + 1) * ((ny + 6) * dr / h2 + 1) * (1.6 * nz * dr / h2 + 1)


def work(case):
    """Bytes: every particle's state (112 B) read and written once a step, or the operator's own inputs and
    outputs; operations: a pair's share of the sums (93; 20 in the wall and filter sums) times the neighbours
    within 2h, and a few hundred a particle in the stress update."""
    soil, wall, cells = _counts(case)
    n = soil + wall
    pairs = soil * 4.0 / 3.0 * math.pi * (2.0 * case["hdr"]) ** 3
    kind = case["kind"]
    if kind in ("march", "dropin"):
        once = dict(bytes=2 * 112 * soil + 24 * wall, flops=2 * 93 * pairs + 400 * soil)
        extra = 112 * n if case.get("reload") else 0
        return dict(bytes=case["steps"] * once["bytes"] + extra, flops=case["steps"] * once["flops"])
    if kind == "search":
        return dict(bytes=16 * n + 8 * n + 8 * cells, flops=10 * n)
    if kind == "pairs":
        return dict(bytes=56 * n + 56 * soil + 8 * cells, flops=93 * pairs)
    if kind == "wall":
        return dict(bytes=44 * soil + 12 * wall + 24 * wall + 8 * cells, flops=20 * 0.1 * pairs)
    return dict(bytes=44 * soil + 24 * soil + 8 * cells, flops=20 * pairs)


# ---------------------------------------------------------- exact, in 64 bits
def _DEV():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _cells(par, x):
    """The particles' cells as whole numbers, in 32-bit arithmetic as the grid's contract has it."""
    c = torch.floor(torch.tensor(0.5, dtype=torch.float32) * x[:, :3].float() * torch.tensor(par.i_h,
                                                                                       dtype=torch.float32))
    return c.long()


def _keys(par, pos):
    """Sort keys: layer, then x, y, z with z fastest."""
    c = _cells(par, pos)
    dims = (par.cell_num_x, par.cell_num_y, par.cell_num_z)
    inside = torch.ones(pos.shape[0], dtype=torch.bool)
    for k in range(3):
        inside &= (c[:, k] >= 0) & (c[:, k] < dims[k])
    layer = (torch.arange(pos.shape[0]) >= par.npb).long() * par.ncell_one_layer
    key = layer + (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
    return torch.where(inside, key, torch.full_like(key, par.ncell_delete))


class _Neighbours:
    """Rows of neighbour indices within a little over 2h, the particle itself left out and as the filler."""

    def __init__(self, par, x, obj, targets, sources, slack):
        dev = x.device
        cut = 2.0 * par.h * (1.0 + slack)
        cell = torch.floor(x[:, :3] / cut).long() + 1
        cell[:, 1] += obj * (int(cell[:, 1].max()) + 3)     # scenarios of an ensemble keep apart
        dim = cell.max(0)[0] + 2
        key = (cell[:, 0] * dim[1] + cell[:, 1]) * dim[2] + cell[:, 2]
        skey, order = torch.sort(key[sources])
        order = sources[order]
        n = targets.numel()
        rows, count = [], torch.zeros(n, dtype=torch.long, device=dev)
        width, self_col = 64, targets
        table = self_col[:, None].repeat(1, width)
        at = torch.arange(n, device=dev)
        xt = x[targets, :3]
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                base = key[targets] + (dx * dim[1] + dy) * dim[2]
                lo = torch.searchsorted(skey, base - 1)
                hi = torch.searchsorted(skey, base + 1, right=True)
                for k in range(int((hi - lo).max())):
                    live = lo + k < hi
                    j = order[torch.where(live, lo + k, torch.zeros_like(lo))]
                    near = live & (j != targets) & (((xt - x[j, :3]) ** 2).sum(1) < cut * cut)
                    if int(count.max()) >= width - 1:
                        table = torch.cat([table, self_col[:, None].repeat(1, 64)], 1)
                        width += 64
                    r = at[near]
                    table[r, count[r]] = j[r]
                    count += near
        self.targets, self.table = targets, table[:, : max(1, int(count.max()))].contiguous()

    def chunks(self, most=12_000_000):
        step = max(1, most // self.table.shape[1])
        for a in range(0, self.targets.numel(), step):
            yield slice(a, a + step), self.targets[a:a + step], self.table[a:a + step]


def _wendland(par, r):
    q = r * par.i_h
    t = torch.clamp(2.0 - q, min=0.0)
    return t, q, par.kernel_normalization_par * t ** 4 * (q + 0.5)


def _exact_wall(par, nb, x, v, s):
    """Boundary stress extrapolated from the soil (Adami), in place in s."""
    g = (par.acc_x, par.acc_y, par.acc_z)
    for _, i, j in nb.chunks():
        d = x[i, None, :3] - x[j][..., :3]
        w = _wendland(par, d.norm(dim=2))[2] * par.m / v[j][..., 3] * (j != i[:, None])
        tot = w.sum(1)
        S = (s[j] * w[..., None]).sum(1)
        acc = (d * w[..., None]).sum(1)
        for k in range(3):
            S[:, k] -= par.rho0 * g[k] * acc[:, k]
        has = tot > 0
        s[i[has]] = S[has] / tot[has, None]


def _exact_pairs(par, nb, x, v, s):
    """(acceleration and density rate, spin, strain rate) of the targets."""
    outs = []
    sig = s / v[:, 3:4] ** 2
    eps = par.artificial_pressure_coefficient
    for _, i, j in nb.chunks(6_000_000):
        d = x[i, None, :3] - x[j][..., :3]
        r2 = (d * d).sum(2)
        t, q, W = _wendland(par, r2.sqrt())
        gr = (par.kernel_gradient_normalization_par * t ** 3)[..., None] * d
        dv = v[i, None, :3] - v[j][..., :3]
        rj = v[j][..., 3]
        drho = (dv * gr).sum(2).sum(1)
        T = sig[i, None] + sig[j]
        if par.viscosity_type == 1:
            vr = torch.clamp((dv * d).sum(2), max=0.0)
            pi = -par.artificial_viscosity_alpha * par.cs * par.h * vr / ((r2 + par.eta) * 0.5 * (v[i, None, 3] + rj))
            T[..., :3] -= pi[..., None]
        if par.artificial_pressure == 1:
            f4 = (W / par.kernel_dr) ** 4
            R = torch.clamp(sig[i, None, :3], min=0.0) + torch.clamp(sig[j][..., :3], min=0.0)
            T[..., :3] -= eps * R * f4[..., None]
        a = torch.stack([T[..., 0] * gr[..., 0] + T[..., 3] * gr[..., 1] + T[..., 4] * gr[..., 2],
                         T[..., 3] * gr[..., 0] + T[..., 1] * gr[..., 1] + T[..., 5] * gr[..., 2],
                         T[..., 4] * gr[..., 0] + T[..., 5] * gr[..., 1] + T[..., 2] * gr[..., 2]], 2).sum(1)
        L = -torch.einsum("nk,nka,nkb->nab", par.m / rj, dv, gr)
        acc = par.m * a + torch.tensor([par.acc_x, par.acc_y, par.acc_z], dtype=x.dtype, device=x.device)
        zero = torch.zeros_like(drho)
        outs.append((torch.cat([acc, par.m * drho[:, None]], 1),
                     0.5 * torch.stack([L[:, 1, 0] - L[:, 0, 1], L[:, 2, 0] - L[:, 0, 2], L[:, 2, 1] - L[:, 1, 2],
                                        zero], 1),
                     torch.stack([L[:, 0, 0], L[:, 1, 1], L[:, 2, 2], 0.5 * (L[:, 0, 1] + L[:, 1, 0]),
                                  0.5 * (L[:, 0, 2] + L[:, 2, 0]), 0.5 * (L[:, 1, 2] + L[:, 2, 1])], 1)))
    return [torch.cat(o) for o in zip(*outs)]


def _exact_smooth(par, nb, x, v, s):
    """Shepard-filtered stress of the soil, the particle itself included."""
    out = []
    w0 = par.kernel_normalization_par * 16.0 * 0.5
    for _, i, j in nb.chunks():
        d = x[i, None, :3] - x[j][..., :3]
        w = _wendland(par, d.norm(dim=2))[2] * par.m / v[j][..., 3] * (j != i[:, None])
        own = w0 * par.m / v[i, 3]
        out.append(((s[j] * w[..., None]).sum(1) + s[i] * own[:, None]) / (w.sum(1) + own)[:, None])
    return torch.cat(out)


def _contract(a, b):
    return (a[:, :3] * b[:, :3]).sum(1) + 2.0 * (a[:, 3:] * b[:, 3:]).sum(1)


def _jaumann(w, s):
    x, y, z = w[:, 0], w[:, 1], w[:, 2]
    return torch.stack([-2.0 * (x * s[:, 3] + y * s[:, 4]), 2.0 * (x * s[:, 3] - z * s[:, 5]),
                        2.0 * (y * s[:, 4] + z * s[:, 5]), x * (s[:, 0] - s[:, 1]) - z * s[:, 4] - y * s[:, 5],
                        y * (s[:, 0] - s[:, 2]) + z * s[:, 3] - x * s[:, 5],
                        z * (s[:, 1] - s[:, 2]) + x * s[:, 4] + y * s[:, 3]], 1)


def _exact_stress(model, mat, dt, w, d, p, ep, s):
    """(stress, pressure, plastic strain) after dt: Drucker-Prager (1) or four-parameter hypoplastic (2)."""
    unit = torch.tensor([1.0, 1.0, 1.0, 0.0, 0.0, 0.0], dtype=s.dtype, device=s.device)
    tr = d[:, :3].sum(1)
    if model == 1:
        K, G, kphi, kpsi, kc = mat
        s = s + dt * (_jaumann(w, s) + (2.0 * G)[:, None] * d + ((K - 2.0 / 3.0 * G) * tr)[:, None] * unit)
        sm = s[:, :3].sum(1) / 3.0
        dev = s - sm[:, None] * unit
        tenf = torch.where(kphi == 0, torch.zeros_like(kc), kc / torch.where(kphi == 0, torch.ones_like(kphi), kphi))
        over = sm - tenf
        cut = over >= 0
        ep = ep + torch.where(cut, over / K * (math.sqrt(2.0) / 3.0), torch.zeros_like(ep))
        sm = torch.where(cut, tenf, sm)
        tau = torch.sqrt(0.5 * _contract(dev, dev))
        f = tau + kphi * sm - kc
        dl = torch.where(f > 0, f / (G + K * kphi * kpsi), torch.zeros_like(f))
        sm = sm - K * kpsi * dl
        small = tau < np.float32(1e-10)
        ratio = torch.where(small, torch.ones_like(tau), (kc - kphi * sm) / torch.where(small, torch.ones_like(tau),
                                                                                       tau))
        dev = torch.where((f > 0)[:, None], dev * ratio[:, None], dev)
        ep = ep + dl * torch.sqrt(1.0 / 3.0 + 2.0 / 9.0 * kpsi * kpsi)
        return dev + sm[:, None] * unit, -sm, ep
    c1, c2, c3, c4, coh = mat
    T = s - torch.clamp(coh, min=0.0)[:, None] * unit
    t1 = T[:, :3].sum(1)
    low = t1.abs() < 4.0
    t1 = torch.where(low, torch.full_like(t1, -4.0), t1)
    T = torch.where(low[:, None], torch.stack([-torch.ones_like(t1), -torch.ones_like(t1), -2.0 * torch.ones_like(t1),
                                               torch.zeros_like(t1), T[:, 4], torch.zeros_like(t1)], 1), T)
    Ts = T - (t1 / 3.0)[:, None] * unit
    nd = torch.sqrt(_contract(d, d))
    s = s + dt * (_jaumann(w, s) + (c1 * t1)[:, None] * d + (c2 * tr + c3 * _contract(T, d) / t1)[:, None] * T
                  + (c4 * nd)[:, None] * (T + Ts))
    pres = s[:, :3].sum(1) / 3.0
    s = s - torch.clamp(pres - coh, min=0.0)[:, None] * unit
    return s, p, ep


def _advance(par, model, mat, dt, st0, half, rates, p_now):
    """(x, v, idep, stress, strain) of the soil `dt` after st0; `half`: the predictor's form of the position."""
    x0, v0, id0, s0, e0 = st0
    a, w, de = rates
    v = v0 + dt * a
    x = x0.clone()
    x[:, :3] += dt * (v[:, :3] if half else 0.5 * (v[:, :3] + v0[:, :3]))
    e = e0 + dt * de
    s, p, ep = _exact_stress(model, mat, dt, w, de, p_now, id0[:, 1], s0)
    if model == 2:
        ep = torch.sqrt(2.0 / 3.0 * _contract(e, e))
    x[:, 3] = p
    i = id0.clone()
    i[:, 1] = ep
    return [x, v, i, s, e]


def _material(c_meta, par, obj):
    one = torch.ones(obj.numel(), dtype=torch.float64, device=obj.device)
    if "materials" in c_meta:
        t = torch.from_numpy(np.asarray(c_meta["materials"])).to(obj.device).double()
        return [t[obj, k] for k in range(5)]
    return [one * getattr(par, "model_par_%d" % k) for k in range(1, 6)]


def _exact_steps(case, c):
    """Whole steps, the particles in their original order throughout."""
    par, dev = c.par, _DEV()
    par.dt = par.cfl * par.h / par.cs
    n, nb = par.np, par.npb
    st = [torch.from_numpy(np.ascontiguousarray(a)).to(dev).double() for a in c.arrays()]
    model, dt = par.constitutive_model, float(par.dt)
    obj = st[2][:, 0].long()
    mat = _material(c.meta, par, obj[nb:])
    apart = obj if "materials" in c.meta else torch.zeros_like(obj)
    wall = torch.arange(nb, device=dev)
    soil = torch.arange(nb, n, device=dev)
    slack = 0.0015 * (case["steps"] + 2)
    of_soil = _Neighbours(par, st[0], apart, soil, torch.arange(n, device=dev), slack)
    of_wall = _Neighbours(par, st[0], apart, wall, soil, slack)
    for _ in range(case["steps"]):
        _exact_wall(par, of_wall, st[0], st[1], st[3])
        rates = _exact_pairs(par, of_soil, st[0], st[1], st[3])
        old = [a[nb:] for a in st]
        new = _advance(par, model, mat, 0.5 * dt, old, True, rates, old[0][:, 3])
        mid = [torch.cat([a[:nb], b]) for a, b in zip(st, new)]
        _exact_wall(par, of_wall, mid[0], mid[1], mid[3])
        rates = _exact_pairs(par, of_soil, mid[0], mid[1], mid[3])
        new = _advance(par, model, mat, dt, old, False, rates, new[0][:, 3])
        st = [torch.cat([a[:nb], b]) for a, b in zip(mid[:4] + [st[4]], new)]
    return dict(pos=st[0], vel=st[1], idep=st[2][:, 1:3], str=st[3], stn=st[4])


def exact(case, seed):
    kind = case["kind"]
    if kind == "search" or case["scene"] == "slope":
        return None     # whole numbers; the adaptive sub-steps of the von Wolffersdorff law have no closed form
    if kind in ("march", "dropin"):
        return _exact_steps(case, _scene(case, seed))
    par, (x, v, i, s, e) = _slot_sorted(case, seed)
    n, nb, dev = par.np, par.npb, x.device
    wall, soil = torch.arange(nb, device=dev), torch.arange(nb, n, device=dev)
    apart = torch.zeros(n, dtype=torch.long, device=dev)
    if kind == "pairs":
        return _exact_pairs(par, _Neighbours(par, x, apart, soil, torch.arange(n, device=dev), 1e-4), x, v, s)
    if kind == "wall":
        _exact_wall(par, _Neighbours(par, x, apart, wall, soil, 1e-4), x, v, s)
        return s
    s[nb:] = _exact_smooth(par, _Neighbours(par, x, apart, soil, soil, 1e-4), x, v, s)
    return s
