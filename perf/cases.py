"""The measured workloads of the dust drag step: what a host code calls between two outputs.

Every case is a pass of a time-stepping run through the public entry points (DeviceDust,
MixedDust, EnsemblePack): a number of cycles from the state of the pass before, with the export
or the cell sort that the run repeats.  The particles are drawn at random from the seed and kept
in cell order, as the periodic cell sort leaves them.

exact() restates the same steps in plain torch, 64 bits, on one global periodic grid (with the
shear-periodic x1 faces of the stratified box), independent of the library's code.  The refined
meshes have none: the general deposit remap and the multilevel prolongation restated in plain
Python take minutes.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

GAMMA = 1.707106781186547          # 1 + 1/sqrt(2)
ETAVK = 0.05                       # the pressure support of the shearing-box set-ups, in c_s
TAUS = (0.01, 0.1, 1.0, 10.0)      # stopping times in units of 1/Omega

# ---------------------------------------------------------------------------------------------
# cases

def listed():
    return [
        # the latency end: 32,768 particles (the plain imex set-up of one small box), where
        # launches and the gaps between them are the cost
        dict(name="mixed_small", kind="mixed", coupling="imex", setup="box", scheme=2, split=True,
             solver=2, nb1=2, nb2=2, nb3=2, nx1=16, nx2=16, nx3=16, ppc=1, nspec=1, cycles=4),
        # a two-dimensional x-z shearing box (streaming instability runs), rotation terms on
        dict(name="mixed_2d", kind="mixed", coupling="imex", setup="si2d", scheme=2, split=True,
             solver=2, nb1=4, nb2=8, nb3=1, nx1=128, nx2=64, nx3=1, ppc=2, nspec=2, cycles=4),
        # blocks of odd sizes, cloud-in-cell weights, plain back-reaction, no defect correction
        dict(name="mixed_ragged", kind="mixed", coupling="imex", setup="box", scheme=1, split=False,
             solver=0, nb1=3, nb2=3, nb3=2, nx1=37, nx2=22, nx3=29, ppc=3, nspec=3, cycles=4),
        # the benchmark's shape at an eighth of its size: 33.5 M particles, 64^3 blocks, 4 species
        # from dt/t_s = 0.01 to 10
        dict(name="mixed_box", kind="mixed", coupling="imex", setup="box", scheme=2, split=True,
             solver=2, nb1=2, nb2=2, nb3=2, nx1=64, nx2=64, nx3=64, ppc=4, nspec=4, cycles=4),
        # a stratified layer with pc2 coupling: shear-periodic x1, outflow x3, a continuous size
        # distribution, every particle within a few scale heights of the midplane
        dict(name="mixed_layer", kind="mixed", coupling="pc2", setup="layer", scheme=2, split=True,
             solver=2, nb1=2, nb2=2, nb3=2, nx1=64, nx2=64, nx3=64, ppc=1, nspec=7, cycles=4),
        # a refined mesh of three levels around a dust clump, blocks of very uneven counts
        dict(name="mixed_refined", kind="refined", form="mixed", root=4, peak=60, cycles=4),
        # an ensemble of independent damping boxes as one pack, cycles replayed from a graph
        dict(name="mixed_ensemble", kind="ensemble", side=24, boxes=32, ppc=3, nspec=3, cycles=10),
        # the FP64 form, rows sorted and then stepped: 4.2 M particles
        dict(name="fp64_box", kind="fp64", coupling="imex", setup="box", scheme=2, split=True,
             solver=2, nb1=2, nb2=2, nb3=2, nx1=32, nx2=32, nx3=32, ppc=4, nspec=4, cycles=4),
        # the FP64 form of a small stratified layer, pc2
        dict(name="fp64_layer", kind="fp64", coupling="pc2", setup="layer", scheme=2, split=True,
             solver=2, nb1=2, nb2=2, nb3=2, nx1=16, nx2=16, nx3=32, ppc=1, nspec=7, cycles=4),
        # refinable clouds on a uniform mesh of 16^3 blocks (FP64, their only form)
        dict(name="cloud_box", kind="cloud", coupling="imex", setup="box", scheme=2, split=True,
             solver=2, nb1=4, nb2=4, nb3=3, nx1=16, nx2=16, nx3=16, ppc=8, nspec=2, cycles=2),
        # refinable clouds over the actual leaves of the refined clump mesh, after the switch and
        # one split pass
        dict(name="cloud_refined", kind="refined", form="cloud", root=4, peak=16, cycles=1),
        # what a run does at an output: the cell sort, the history row, the science fields and the
        # self-gravity transfer both ways
        dict(name="output", kind="output", coupling="imex", setup="box", scheme=2, split=True,
             solver=2, nb1=3, nb2=2, nb3=3, nx1=32, nx2=32, nx3=32, ppc=3, nspec=2, cycles=1),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mixed", "mixed", "mixed", "fp64", "fp64", "cloud", "refined", "ensemble",
                       "output"])
    if kind == "refined":
        form = rng.choice(["mixed", "fp64", "cloud"])
        return dict(kind=kind, form=form, root=rng.choice([3, 4, 4]), peak=_logint(rng, 4, 24),
                    cycles=rng.randint(1, 3))
    if kind == "ensemble":
        return dict(kind=kind, side=_logint(rng, 16, 48), boxes=rng.randint(2, 24),
                    ppc=rng.randint(1, 4), nspec=rng.randint(1, 4), cycles=rng.randint(4, 12))
    c = dict(kind=kind, coupling="imex", setup="box", scheme=2, split=True, solver=2)
    c["nspec"] = rng.randint(1, 4)
    c["ppc"] = rng.randint(1, 4)
    if kind in ("mixed", "fp64"):
        c["setup"] = rng.choice(["box", "box", "si2d", "layer"])
        c["scheme"] = rng.choice([2, 2, 1, 0])
        c["split"] = rng.random() < 0.6
        c["solver"] = rng.choice([0, 2, 2, 3])
    if c["setup"] == "layer":
        # (an even number of cells in x3 around the midplane, at least six scale heights each way)
        c.update(coupling="pc2", nspec=rng.randint(1, 7), ppc=1, scheme=2, split=True, solver=2)
        c.update(nb1=2, nb2=rng.randint(1, 3), nb3=2, nx1=rng.randint(10, 40),
                 nx2=rng.randint(10, 40), nx3=rng.randint(24, 48))
    elif c["setup"] == "si2d":
        c.update(nb1=rng.randint(1, 4), nb2=rng.randint(1, 4), nb3=1, nx1=_logint(rng, 16, 160),
                 nx2=_logint(rng, 16, 160), nx3=1)
    else:
        top = {"mixed": 48, "fp64": 32, "cloud": 20, "output": 32}[kind]
        c.update(nb1=rng.randint(1, 3), nb2=rng.randint(1, 3), nb3=rng.randint(1, 3),
                 nx1=_logint(rng, 9, top), nx2=_logint(rng, 9, top), nx3=_logint(rng, 9, top))
        if kind == "cloud":
            c["ppc"] = rng.randint(2, 8)
    c["cycles"] = 1 if kind == "output" else rng.randint(2, 4)
    # no drawn case beyond the largest listed one of its kind
    most = {"mixed": 1.0e8, "fp64": 1.2e7, "cloud": 6.0e6, "output": 3.5e6}[kind]
    while Setup(c).npart * c["cycles"] > most:
        if c["cycles"] > 1:
            c["cycles"] -= 1
        elif c["nspec"] > 1:
            c["nspec"] -= 1
        else:
            c["ppc"] -= 1
    return c


# ---------------------------------------------------------------------------------------------
# set-ups, in plain torch

class Setup:
    """The box, the time step and the physics of a case (plain numbers)."""

    def __init__(self, case):
        self.N = (case["nb1"] * case["nx1"], case["nb2"] * case["nx2"], case["nb3"] * case["nx3"])
        self.nb = (case["nb1"], case["nb2"], case["nb3"])
        self.nx = (case["nx1"], case["nx2"], case["nx3"])
        self.setup = case["setup"]
        self.three_d = self.N[2] > 1
        self.layer = self.setup == "layer"
        self.rot = self.setup != "box"           # rotation and shear terms
        self.time = 3.7 if self.layer else 0.0
        if self.layer:
            self.dx = 0.00625
            self.taus = [10.0 ** (-3.0 + 3.0 * (s + 0.5) / case["nspec"])
                         for s in range(case["nspec"])]
            self.eps = [0.01 / case["nspec"]] * case["nspec"]
            self.hp = min(0.02, self.N[2] * self.dx / 14.0)
            self.dt = 0.3 * self.dx / (1.0 + 1.5 * 0.5 * self.N[0] * self.dx)
        else:
            self.taus = list(TAUS[:case["nspec"]]) if case["nspec"] > 1 else [0.1]
            self.eps = [0.5] * case["nspec"]
            if self.setup == "si2d":
                self.dx = 0.02
                self.dt = 0.3 * self.dx / 1.05
            else:
                self.dt = 0.1
                self.dx = self.dt * 1.05 / 0.3
        self.L = [self.N[0] * self.dx, self.N[1] * self.dx,
                  self.N[2] * self.dx if self.three_d else 1.0]
        self.lo = [-0.5 * x for x in self.L]
        self.hi = [0.5 * x for x in self.L]
        self.vol = self.dx ** 3 if self.three_d else self.dx ** 2
        self.ncell = self.N[0] * self.N[1] * self.N[2]
        self.npart = self.ncell * case["ppc"] * case["nspec"]
        self.phys = dict(scheme=case["scheme"], drag_solver=case["solver"], back_reaction=True,
                         consistent_gas=case["split"], shearing_box=self.rot,
                         stratified=self.layer, qshear=1.5, omega0=1.0)


def _drift(tau):
    """The drift of a trace species in the shearing box (radial, azimuthal)."""
    return -2.0 * ETAVK * tau / (1.0 + tau * tau), -ETAVK / (1.0 + tau * tau)


def _inputs(case, seed, device="cuda"):
    """Positions, velocities (3, N), stopping times, masses, species, blocks, in cell order, and
    the gas momentum (3, N3, N2, N1) at density 1, from the seed."""
    S = Setup(case)
    g = torch.Generator(device=device)
    g.manual_seed(int(seed) * 7919 + 11)
    f64 = dict(device=device, dtype=torch.float64)
    n, per = S.npart, S.ncell * case["ppc"]
    sp = torch.arange(n, device=device, dtype=torch.int64) // per
    x = torch.empty((3, n), **f64)
    for a in range(3):
        u = torch.rand(n, generator=g, **f64)
        x[a] = S.lo[a] + u * S.L[a]
        del u
    if not S.three_d:
        x[2] = 0.0
    if S.layer:
        z = S.hp * torch.randn(n, generator=g, **f64)
        x[2] = z.clamp(-6.0 * S.hp, 6.0 * S.hp)
        del z
    # cell order: block, then k, j, i inside the block
    key = torch.zeros(n, device=device, dtype=torch.int64)
    cell = []
    for a in range(3):
        c = torch.floor((x[a] - S.lo[a]) / (S.L[a] / S.N[a])).long().clamp_(0, S.N[a] - 1)
        cell.append(c)
    blk = ((cell[2] // S.nx[2]) * S.nb[1] + cell[1] // S.nx[1]) * S.nb[0] + cell[0] // S.nx[0]
    key = ((blk * S.nx[2] + cell[2] % S.nx[2]) * S.nx[1] + cell[1] % S.nx[1]) * S.nx[0] \
        + cell[0] % S.nx[0]
    del cell
    order = torch.sort(key, stable=True).indices
    del key
    x = x[:, order].contiguous()
    sp = sp[order]
    blk = blk[order]
    del order
    taus = torch.tensor(S.taus, **f64)
    if S.layer:
        # each particle its own stopping time inside its bin
        w = math.log(1000.0) / case["nspec"]
        ts = taus[sp] * torch.exp((torch.rand(n, generator=g, **f64) - 0.5) * w)
    else:
        ts = taus[sp]
    m = torch.tensor([e * S.ncell * S.vol * (1.0 if S.three_d else S.L[2]) / per for e in S.eps],
                     **f64)[sp]
    v = torch.empty((3, n), **f64)
    for a in range(3):
        v[a] = 1e-3 * torch.randn(n, generator=g, **f64)
    d = torch.tensor([_drift(t) for t in S.taus], **f64)
    v[0] += d[sp, 0]
    v[1 if S.three_d else 2] += d[sp, 1]
    N1, N2, N3 = S.N
    mom = 1e-3 * (2.0 * torch.rand((3, N3, N2, N1), generator=g, **f64) - 1.0)
    mom[1 if S.three_d else 2] -= ETAVK
    return S, x, v, ts, m, sp, blk, mom


@functools.lru_cache(maxsize=64)
def _mesh(N, nx, lo, hi, x3bc, shear):
    from athenak_b200.mesh import uniform_mesh
    return uniform_mesh(N, nx, 2, lo, hi, x3bc=x3bc, shear_x1=shear)


def _to_blocks(S, f):
    """(V, N3, N2, N1) -> (nmb, V, nx3, nx2, nx1), blocks x1 fastest."""
    V = f.shape[0]
    f = f.reshape(V, S.nb[2], S.nx[2], S.nb[1], S.nx[1], S.nb[0], S.nx[0])
    return f.permute(1, 3, 5, 0, 2, 4, 6).reshape(-1, V, S.nx[2], S.nx[1], S.nx[0])


def _device_dust(case, seed):
    from athenak_b200.drag import DeviceDust
    S, x, v, ts, m, sp, blk, mom = _inputs(case, seed)
    ms = _mesh(S.N, S.nx, tuple(S.lo), tuple(S.hi), 2 if S.layer else 0, S.layer)
    dev = DeviceDust.empty(ms, S.npart, S.phys, nspecies=case["nspec"])
    pr, pi = dev.t["pr"], dev.t["pi"]
    for a in range(3):
        pr[2 * a], pr[2 * a + 6] = x[a], x[a]
        pr[2 * a + 1], pr[2 * a + 7] = v[a], v[a]
    pr[15], pr[16] = ts, m
    pi[0], pi[2] = blk.int(), sp.int()
    pi[1] = torch.arange(S.npart, device=pi.device, dtype=torch.int32)
    act = ms.active(dev.t["u0"])
    act[:, 0] = 1.0
    act[:, 1:4] = _to_blocks(S, mom)
    dev.t["u0"][:, 0] = 1.0
    if S.layer:
        dev.set_time(S.time)
    dev.init_gas_ghosts()
    return S, dev, ms


# ---------------------------------------------------------------------------------------------
# the refined clump mesh

def _clump_refine(e, c):
    r = math.sqrt(sum(x * x for x in c))
    return r < (0.33 if e == 0 else 0.16)


@functools.lru_cache(maxsize=4)
def _clump_mesh(root):
    from athenak_b200.amr import build_dep_plan, leaf_tables, refined_mesh
    ms = refined_mesh((root,) * 3, (16, 16, 16), 2, (-0.5,) * 3, (0.5,) * 3, refine=_clump_refine)
    return ms, build_dep_plan(ms, 0), leaf_tables(ms)


def _clump(case, seed, device="cuda"):
    """Point particles of two species around a Gaussian clump on the refined mesh, in cell
    order: 1 + floor(peak exp(-r^2 / 2 sigma^2)) of each species in every cell."""
    from athenak_b200.drag import DeviceDust
    ms, plan, _ = _clump_mesh(case["root"])
    g = torch.Generator(device=device)
    g.manual_seed(int(seed) * 7919 + 13)
    f64 = dict(device=device, dtype=torch.float64)
    nx, nmb, sigma = 16, ms.nmb, 0.05
    mb = torch.from_numpy(np.ascontiguousarray(ms.mb_size)).to(device)
    c = torch.arange(nmb * nx ** 3, device=device)
    cm, ci, cj, ck = c // nx ** 3, c % nx, (c // nx) % nx, (c // nx ** 2) % nx
    idx = torch.stack([ci, cj, ck], 1).double()
    dx = mb[cm, 6:9]
    r2 = ((mb[cm, 0:3] + (idx + 0.5) * dx) ** 2).sum(1)
    bump = torch.exp(-r2 / (2.0 * sigma ** 2))
    cnt = 1 + torch.floor(case["peak"] * bump).long()
    npart = 2 * int(cnt.sum())
    dev = DeviceDust.empty(ms, npart, dict(scheme=2, drag_solver=0, consistent_gas=True,
                                           back_reaction=True), nspecies=2)
    pr, pi = dev.t["pr"], dev.t["pi"]
    # (clouds at fixed places: the number of pieces the split appends follows from them; their
    # velocities are the seed's)
    gx = g
    if case["form"] == "cloud":
        gx = torch.Generator(device=device)
        gx.manual_seed(13)
    cell2 = torch.repeat_interleave(torch.arange(2 * c.numel(), device=device),
                                    cnt.repeat_interleave(2))
    p, sp = cell2 // 2, cell2 % 2
    for a in range(3):
        # (kept a hair inside the cell: a draw at its upper edge would round onto the next one)
        u = torch.rand(npart, generator=gx, **f64).clamp_(1e-9, 1.0 - 1e-9)
        pr[2 * a] = mb[cm[p], a] + (idx[p, a] + u) * dx[p, a]
        pr[2 * a + 6] = pr[2 * a]
        pr[2 * a + 1] = 1e-2 * torch.randn(npart, generator=g, **f64)
        pr[2 * a + 7] = pr[2 * a + 1]
    pr[15] = torch.tensor([0.1, 1.0], **f64)[sp]
    vol = dx.prod(1)
    pr[16] = (0.5 * (0.01 + 100.0 * bump) * vol / cnt)[p]
    pi[0], pi[2] = cm[p].int(), sp.int()
    pi[1] = torch.arange(npart, device=device, dtype=torch.int32)
    u0 = dev.t["u0"]
    u0[:, 0] = 1.0
    u0[:, 1:4] = 1e-3 * (2.0 * torch.rand(u0[:, 1:4].shape, generator=g, **f64) - 1.0)
    dev.set_dep_plan(plan)
    dev.ghost_copy_ml("u0", 4)
    dt = 0.3 * float(ms.mb_size[:, 6].min()) / 1.05
    return dev, ms, dt


# ---------------------------------------------------------------------------------------------
# the ensemble

def _boxes(case, seed):
    """(taus, eps) of every box, log-uniform over the ensemble's ranges."""
    rng = np.random.default_rng(int(seed) * 7919 + 17)
    ns = case["nspec"]
    return [(tuple(float(t) for t in np.exp(rng.uniform(math.log(1e-2), math.log(10.0), ns))),
             tuple(float(t) for t in np.exp(rng.uniform(math.log(0.1), math.log(4.0), ns))))
            for _ in range(case["boxes"])]


# ---------------------------------------------------------------------------------------------
# prepare and run

class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, s.kind = case, case["kind"]
    if s.kind == "ensemble":
        from athenak_b200.ensemble import Box, EnsemblePack
        s.pack = EnsemblePack(case["side"], [Box(case["side"], t, e, case["ppc"])
                                             for t, e in _boxes(case, seed)])
        s.pack.step(1)                    # the first cycle, then the captured graph is kept
        s.dev, s.ms, s.n = s.pack.dev, s.pack.ms, s.pack.npart
        return s
    if s.kind == "refined":
        s.dev, s.ms, s.dt = _clump(case, seed)
        if case["form"] == "mixed":
            from athenak_b200.mixed import MixedDust
            s.mx = MixedDust(dev=s.dev)
        elif case["form"] == "cloud":
            from athenak_b200 import capi
            lt = _clump_mesh(case["root"])[2]
            s.dev.set_leaf_tables(lt)
            s.dev.cloud_instant_switch(0)
            s.dev.cloud_split_p1(capi.split_params(max_level=lt.nlev), int(s.dev.npart))
        s.n = s.dev.npart
        return s
    S, s.dev, s.ms = _device_dust(case, seed)
    s.dt, s.n = S.dt, S.npart
    if s.kind == "mixed":
        from athenak_b200.mixed import MixedDust
        s.mx = MixedDust(dev=s.dev)
    if s.kind == "output":
        s.force = torch.empty(s.ms.field_shape(3), device="cuda", dtype=torch.float64)
        s.force.copy_(s.dev.t["u0"][:, 1:4])
    return s


def _rows(s):
    """The particle rows and the gas of the active cells, by what they hold."""
    pr, pi = s.dev.t["pr"][:, :s.n], s.dev.t["pi"][:, :s.n]
    return {"x": pr[0:6:2], "v": pr[1:6:2], "x1": pr[6:12:2], "v1": pr[7:12:2], "rate": pr[12:15],
            "block": pi[0], "gas": s.ms.active(s.dev.t["u0"])}


def run(s):
    case = s.case
    n = case["cycles"]
    if s.kind == "ensemble":
        s.pack.step(n)
        s.pack.mx.export()
        return _rows(s)
    if s.kind == "refined":
        if case["form"] == "mixed":
            for _ in range(n):
                s.mx.imex_cycle(s.dt)
            s.mx.export()
        elif case["form"] == "cloud":
            for _ in range(n):
                s.dev.cloud_refined_imex_cycle(s.dt)
        else:
            for _ in range(n):
                s.dev.refined_imex_cycle(s.dt)
        return _rows(s)
    if s.kind == "output":
        s.dev.sort_by_cell()
        row = s.dev.phst()
        sci = s.dev.point_science_fields()
        rho = s.dev.point_gravity_density()
        acc = s.dev.point_gravity_gather(s.force)
        out = _rows(s)
        return {"x": out["x"], "v": out["v"], "block": out["block"], "row": row,
                "science": s.ms.active(sci), "density": s.ms.active(rho), "acc": acc}
    if s.kind == "mixed":
        for _ in range(n):
            if case["coupling"] == "imex":
                s.mx.imex_cycle(s.dt)
            else:
                chi = s.mx.pc2_cycle(s.dt)
        s.mx.export()
    elif s.kind == "fp64":
        s.dev.sort_by_cell()
        for _ in range(n):
            if case["coupling"] == "imex":
                s.dev.imex_cycle(s.dt)
            else:
                chi = s.dev.pc2_cycle(s.dt)
    else:
        s.dev.sort_by_cell()
        for _ in range(n):
            s.dev.cloud_imex_cycle(s.dt)
    out = _rows(s)
    if case["coupling"] == "pc2":
        out["chi"] = chi
    return out


# ---------------------------------------------------------------------------------------------
# work: the state read and written once per cycle, the weights' multiply-adds

def _counts(case):
    if case["kind"] == "ensemble":
        c = case["boxes"] * case["side"] ** 3
        return c, c * case["ppc"] * case["nspec"]
    if case["kind"] == "refined":
        ms = _clump_mesh(case["root"])[0]
        nx = 16
        o = np.arange(nx) + 0.5
        r2 = [(ms.mb_size[:, a, None] + o * ms.mb_size[:, 6 + a, None]) ** 2 for a in range(3)]
        r2 = r2[2][:, :, None, None] + r2[1][:, None, :, None] + r2[0][:, None, None, :]
        cnt = 1 + np.floor(case["peak"] * np.exp(-r2 / (2.0 * 0.05 ** 2)))
        return ms.nmb * nx ** 3, int(2 * cnt.sum())
    S = Setup(case)
    return S.ncell, S.npart


def work(case):
    cells, parts = _counts(case)
    n = case["cycles"]
    if case["kind"] == "output":
        # rows in and out of the sort, the sums and three transfers over x, v, m
        return {"bytes": float(parts * (2 * 156 + 56 + 56 + 32 + 32 + 24) + cells * 8 * (1 + 4 + 1 + 3)),
                "flops": float(parts * 27 * 2 * (1 + 4 + 1 + 3))}
    mixed = case["kind"] in ("mixed", "ensemble") or case.get("form") == "mixed"
    real = 4 if mixed else 8
    # per cycle: x, v, rate, t_s, m and the owner read; x, v, their registers, rate and the owner
    # written; the gas (4 values) read and written
    b = parts * n * ((11 + 15) * real + 8) + cells * n * 64
    if mixed:
        b += parts * (15 * 8 + 4)                      # the export to the FP64 rows
    elif case["kind"] in ("fp64", "cloud"):
        b += parts * 2 * 156                           # the sort
    dep = 27 if (case.get("nx3", 16) > 1) else 9
    pc2 = case.get("coupling") == "pc2"
    solver = 2 if case["kind"] == "ensemble" else case.get("solver", 0)
    sweeps = {0: 0, 2: 1, 3: 2}[solver]
    # values gathered and deposited per particle and cycle
    vals = (3 + 4 + 3 + 3) if pc2 else 2 * (4 + 6 * sweeps + 6)
    return {"bytes": float(b), "flops": float(parts * n * vals * dep * 2)}


def tolerance(case):
    mixed = case["kind"] in ("mixed", "ensemble") or case.get("form") == "mixed"
    if not mixed:
        # FP64 sums in another order: 5e-15 (2-norm) and 4e-13 (largest) between two runs
        return {"rel": 1e-12, "max": 1e-10, "differ": 1e-6}
    if case.get("coupling") == "pc2":
        # FP32 weights, gathers and kicks: 4e-5 against exact(), the rates of the stiffest bins
        return {"rel": 2e-4, "max": 0.05, "differ": 1e-5}
    if not case.get("split", True):
        # 1e-6 against exact()
        return {"rel": 5e-6, "max": 1e-3, "differ": 1e-5}
    # the consistent split is a step function of the position: a particle within FP32 rounding
    # of a cell face takes its neighbour cell's share (5e-4 of the rates against exact())
    return {"rel": 2e-3, "max": 0.9, "differ": 1e-5}


# ---------------------------------------------------------------------------------------------
# exact: the same steps in plain torch, 64 bits

class Plain:
    """Particles on one global grid of N cells: periodic in x2, in x1 (or shear-periodic) and in
    x3 (the stratified layer never reaches its x3 faces).  Fields are (3, N3, N2, N1)."""

    def __init__(self, N, dx, lo, L, scheme, solver, split, x, v, ts, m, mom, shear=None,
                 rot=False, strat=False):
        self.N, self.dx, self.lo, self.L = N, dx, lo, L
        self.scheme, self.solver, self.split = scheme, solver, split
        self.three_d = N[2] > 1
        self.vol = dx ** 3 if self.three_d else dx * dx
        self.x, self.v, self.ts, self.m = x.clone(), v.clone(), ts, m
        self.x1, self.v1 = x.clone(), v.clone()
        self.R = torch.zeros_like(v)
        self.rho, self.mom = torch.ones_like(mom[0]), mom.clone()
        self.dmom = torch.zeros_like(mom)
        self.shear, self.rot, self.strat = shear, rot, strat
        self.dev = x.device

    # -- weights: the anchor cell of every particle and its three weights along each axis
    def _axis(self, xa, a):
        c = (xa - self.lo[a]) / self.dx
        i = torch.floor(c)
        d = c - (i + 0.5)
        if self.scheme == 0:
            w = (None, torch.ones_like(d), None)
        elif self.scheme == 1:
            w = ((-d).clamp(min=0.0), 1.0 - d.abs(), d.clamp(min=0.0))
        else:
            w = (0.5 * (0.5 - d) ** 2, 0.75 - d * d, 0.5 * (0.5 + d) ** 2)
        return i.long(), w

    def place(self, x):
        self.ax = [self._axis(x[a], a) for a in range(3 if self.three_d else 2)]

    def _stencil(self):
        """(weight, flat index into the padded grid) of every stencil cell."""
        N1, N2, N3 = self.N
        (i, wx), (j, wy) = self.ax[0], self.ax[1]
        for c in ((-1, 0, 1) if self.three_d else (0,)):
            if self.three_d:
                k, wz = self.ax[2]
                if wz[c + 1] is None:
                    continue
                kk = k + c
                kk = kk.clamp(0, N3 - 1) if self.shear else kk % N3
            for b in (-1, 0, 1):
                if wy[b + 1] is None:
                    continue
                jj = (j + b) % N2
                w2 = wy[b + 1] * wz[c + 1] if self.three_d else wy[b + 1]
                row = (kk * N2 + jj) * (N1 + 4) if self.three_d else jj * (N1 + 4)
                for a in (-1, 0, 1):
                    if wx[a + 1] is None:
                        continue
                    yield w2 * wx[a + 1], row + (i + a + 2), (a, b, c)

    # -- x1 padding (two ghost columns) and its transpose for deposits
    def pad(self, f):
        g0, g1 = f[..., -2:], f[..., :2]
        if self.shear:
            yun, _ = self.shear
            dy = self.dx
            joff = int(yun / dy)
            eps = math.fmod(yun, dy) / dy
            g0 = self._remap(g0, joff, eps)
            g1 = self._remap(g1, -joff, -eps)
        return torch.cat([g0, f, g1], dim=-1)

    @staticmethod
    def _remap(g, joff, eps):
        g = torch.roll(g, joff, dims=-2)                      # row J takes row J - joff
        at = lambda t: torch.roll(g, -t, dims=-2)             # noqa: E731  row r + t

        def flux(q):
            a, b, c, d = at(q - 2), at(q - 1), at(q), at(q + 1)
            l, r = (b - a, c - b) if eps > 0.0 else (c - b, d - c)
            p = l * r
            s = torch.where(p <= 0.0, torch.zeros_like(p), 2.0 * p / (l + r))
            return eps * (b + 0.5 * (1.0 - eps) * s) if eps > 0.0 else eps * (c - 0.5 * (1.0 + eps) * s)
        return g - (flux(1) - flux(0))

    def fold(self, f):
        """(.., N1 + 4) deposits -> (.., N1): the ghost columns into the other face's strip."""
        out = f[..., 2:-2].clone()
        lo, hi = f[..., :2], f[..., -2:]
        if self.shear:
            sh = self.shear[1] / self.dx
            lo, hi = self._shift(lo, -sh), self._shift(hi, sh)
        out[..., -2:] += lo
        out[..., :2] += hi
        return out

    @staticmethod
    def _shift(g, s):
        k = math.floor(s)
        f = s - k
        return (1.0 - f) * torch.roll(g, k, dims=-2) + f * torch.roll(g, k + 1, dims=-2)

    def gather(self, f):
        p = self.pad(f).reshape(f.shape[0], -1)
        out = [torch.zeros_like(self.ts) for _ in range(f.shape[0])]
        for w, at, _ in self._stencil():
            for q in range(f.shape[0]):
                out[q] += w * p[q][at]
        return out

    def deposit(self, vals):
        N1, N2, N3 = self.N
        f = torch.zeros((len(vals), N3 * N2 * (N1 + 4)), device=self.dev, dtype=torch.float64)
        for w, at, _ in self._stencil():
            for q, val in enumerate(vals):
                f[q].index_add_(0, at, w * val)
        return self.fold(f.reshape(len(vals), N3, N2, N1 + 4))

    def centre(self):
        N1, N2, N3 = self.N
        i, j = self.ax[0][0] % N1, self.ax[1][0] % N2
        return ((self.ax[2][0] % N3) * N2 + j) * N1 + i if self.three_d else j * N1 + i

    # -- routing: wrap into the box, the register with the position
    def route(self):
        lo, L = self.lo, self.L
        if self.shear:
            ysh = self.shear[1]
            out = (self.x[0] < lo[0]).double() - (self.x[0] >= lo[0] + L[0]).double()
            y = self.x[1] - out * ysh
            y = torch.where((out != 0) & (y < lo[1]), y + L[1], y)
            y = torch.where((out != 0) & (y >= lo[1] + L[1]), y - L[1], y)
            y = torch.where(out != 0, y, self.x[1])
            self.x1[1] += y - self.x[1]
            self.x[1] = y
            self.x[0] += out * L[0]
            self.x1[0] += out * L[0]
        for a in range(3 if self.three_d and not self.shear else 2):
            if a == 0 and self.shear:
                continue
            s = L[a] * ((self.x[a] < lo[a]).double() - (self.x[a] >= lo[a] + L[a]).double())
            self.x[a] += s
            self.x1[a] += s

    def _force(self):
        f = [0.0, 0.0, 0.0]
        if self.rot and self.three_d:
            f = [2.0 * self.v[1], -0.5 * self.v[0], -self.x[2] if self.strat else 0.0]
        elif self.rot:
            f = [2.0 * self.v[2], 0.0, -0.5 * self.v[0]]
        return f

    def imex(self, dt, cloud=False):
        g = GAMMA
        t2 = (2.0 * g - 1.0) / (2.0 * g * g)
        atw = (1.0 - 2.0 * g * g) / 2.0 / g * dt
        a_dt = g * dt
        for g0, g1, beta, stage in ((1.0, 0.0, g * dt, 1), (t2, 1.0 - t2, dt / (2.0 * g), 2)):
            if stage == 1:
                self.x1, self.v1 = self.x.clone(), self.v.clone()
                u1 = (self.rho.clone(), self.mom.clone())
            else:
                self.rho = g0 * self.rho + g1 * u1[0]
                self.mom = g0 * self.mom + g1 * u1[1] + atw * self.dmom
            f = self._force()
            vo, xo = self.v.clone(), self.x.clone()
            for a in range(3):
                self.v[a] = g0 * vo[a] + g1 * self.v1[a] + beta * f[a]
                if stage == 2:
                    self.v[a] += atw * self.R[a]
                vd = vo[a] - (1.5 * xo[0] if (a == 1 and self.rot and self.three_d) else 0.0)
                if a < 2 or self.three_d:
                    self.x[a] = g0 * xo[a] + g1 * self.x1[a] + beta * vd
            del vo, xo, f
            self.route()
            self.place(self.x)
            c = a_dt / (self.ts + a_dt)
            q = self.m * c / self.vol
            dep = self.deposit([q, q * self.v[0], q * self.v[1], q * self.v[2]])
            Q, P = dep[0], dep[1:]
            us = (self.mom + P) / (self.rho + Q)
            for _ in range({0: 0, 2: 1, 3: 2}[self.solver]):
                ub = self._gather_moments(us) if cloud else self.gather(us)
                res = self.deposit([q * ub[0], q * ub[1], q * ub[2]])
                us = us + (self.mom + P - res - self.rho * us) / (self.rho + Q)
            ub = self._gather_moments(us) if cloud else self.gather(us)
            dv = [c * (ub[a] - self.v[a]) for a in range(3)]
            for a in range(3):
                self.v[a] += dv[a]
                self.R[a] = dv[a] / a_dt
            mv = -self.m / self.vol
            dm = self.deposit([mv * d for d in dv])
            gq = self.rho * us - self.mom
            r = (dm - gq) / (self.rho + Q)
            if cloud:
                self.mom += gq + self.rho * r
                self.dmom = (gq + self.rho * r) / a_dt
                rv = self.gather(r)
                for a in range(3):
                    self.v[a] += c * rv[a]
                    self.R[a] += c * rv[a] / a_dt
            elif self.split:
                cc = self.centre()
                qt = torch.zeros(Q.numel(), device=self.dev, dtype=torch.float64)
                qt.index_add_(0, cc, q)
                qt = qt.reshape(Q.shape)
                has = qt > 0.0
                dg = torch.where(has, gq + self.rho * r, dm)
                self.mom += dg
                self.dmom = dg / a_dt
                share = torch.where(has, r * Q / torch.where(has, qt, torch.ones_like(qt)),
                                    torch.zeros_like(r)).reshape(3, -1)
                for a in range(3):
                    d = c * share[a][cc]
                    self.v[a] += d
                    self.R[a] += d / a_dt
            else:
                self.mom += dm
                self.dmom = dm / a_dt

    # -- the clouds' linear gather: the hat's first moments with central differences
    def _gather_moments(self, us):
        N1, N2, N3 = self.N
        g = [us] + [torch.roll(us, -1, d) - torch.roll(us, 1, d) for d in (3, 2, 1)]
        g = [self.pad(t).reshape(3, -1) for t in g]

        def mom1(s):
            # the antiderivative of the hat's first moment, from the centre
            s = s.clamp(-1.0, 1.0)
            return 0.5 * s * s - s.abs() ** 3 / 3.0
        M = []
        for a, (i, _) in enumerate(self.ax):
            t = (self.x[a] - self.lo[a]) / self.dx - i.double()      # place in the cell, 0..1
            M.append([(o + 1 - t, mom1(o + 1 - t) - mom1(o - t), t - o - 0.5) for o in (-1, 0, 1)])
        W = [w for _, w in self.ax]
        out = [torch.zeros_like(self.ts) for _ in range(3)]
        for w, at, (a, b, c) in self._stencil():
            idx = (a + 1, b + 1, c + 1)
            co = []
            for d in range(3):
                e = [W[q][idx[q]] for q in range(3)]
                e[d] = M[d][idx[d]][1]
                co.append(0.5 * (e[0] * e[1] * e[2] + M[d][idx[d]][2] * w))
            for q in range(3):
                out[q] += w * g[0][q][at] + co[0] * g[1][q][at] + co[1] * g[2][q][at] \
                    + co[2] * g[3][q][at]
        return out

    def pc2(self, dt):
        h = 0.5 * dt
        self.x1, self.v1 = self.x.clone(), self.v.clone()
        rho1, mom1 = self.rho.clone(), self.mom.clone()
        self.place(self.x)
        ug = self.gather(self.mom / self.rho)
        rate = self.m / (self.ts * self.vol)
        dep = self.deposit([-dt * rate * (ug[0] - self.v[0]), -dt * rate * (ug[1] - self.v[1]),
                            -dt * rate * (ug[2] - self.v[2]), rate])
        chi = dt * dep[3] / self.rho
        dep = dep[:3] / chi.clamp(min=1.0)
        self.mom = self.mom + dep
        us = (mom1 + self.mom) / (rho1 + self.rho)
        self.mom = 0.5 * (self.mom + mom1)
        x0, v0 = self.x1, self.v1
        sh3 = self.rot and self.three_d
        xh = x0 + h * v0
        if sh3:
            xh[1] -= h * 1.5 * x0[0]
        if not self.three_d:
            xh[2] = x0[2]
        xg = xh.clone()
        if sh3:
            xg[1] += 1.5 * xh[0] * h
        self.place(xg)
        ug = self.gather(us)
        lam = h / self.ts
        aa = 1.0 + lam
        r = [v0[a] + lam * ug[a] for a in range(3)]
        if sh3:
            det = aa * aa + h * h
            vh = [(aa * r[0] + 2.0 * h * r[1]) / det, (aa * r[1] - 0.5 * h * r[0]) / det,
                  (r[2] - (h * xh[2] if self.strat else 0.0)) / aa]
        elif self.rot:
            det = aa * aa + h * h
            vh = [(aa * r[0] + 2.0 * h * r[2]) / det, r[1] / aa, (aa * r[2] - 0.5 * h * r[0]) / det]
        else:
            vh = [t / aa for t in r]
        vh = torch.stack(vh)
        self.v = 2.0 * vh - v0
        vd = vh.clone()
        if sh3:
            vd[1] -= 1.5 * xh[0]
        xn = x0 + dt * vd
        if not self.three_d:
            xn[2] = x0[2]
        self.R = torch.stack([dt * (ug[a] - vh[a]) / self.ts for a in range(3)])
        mv = -self.m / self.vol
        dm = self.deposit([mv * self.R[a] for a in range(3)])
        self.x, self.x1 = xn, xh
        self.route()
        self.mom = self.mom + dm - 0.5 * dep
        return chi.max()


def _result(p, S, chi=None):
    cell = [torch.floor((p.x[a] - S.lo[a]) / S.dx).long().clamp(0, S.N[a] - 1)
            if S.N[a] > 1 else torch.zeros_like(p.ts, dtype=torch.int64) for a in range(3)]
    blk = ((cell[2] // S.nx[2]) * S.nb[1] + cell[1] // S.nx[1]) * S.nb[0] + cell[0] // S.nx[0]
    out = {"x": p.x, "v": p.v, "x1": p.x1, "v1": p.v1, "rate": p.R, "block": blk.int(),
           "gas": _to_blocks(S, torch.cat([p.rho[None], p.mom]))}
    if chi is not None:
        out["chi"] = chi
    return out


def exact(case, seed):
    if case["kind"] == "refined":
        return None
    if case["kind"] == "ensemble":
        return _exact_ensemble(case, seed)
    S, x, v, ts, m, sp, blk, mom = _inputs(case, seed)
    shear = None
    if S.layer:
        y = 1.5 * S.L[0] * S.time
        shear = (y, math.fmod(y, S.L[1]))
    p = Plain(S.N, S.dx, S.lo, S.L, case["scheme"], case["solver"], case["split"], x, v, ts, m,
              mom, shear, S.rot, S.layer)
    if case["kind"] == "output":
        return _exact_output(p, S, x, v, m, blk, mom)
    chi = None
    for _ in range(case["cycles"]):
        if case["coupling"] == "pc2":
            chi = p.pc2(S.dt)
        else:
            p.imex(S.dt, cloud=case["kind"] == "cloud")
    out = _result(p, S, chi)
    if case["kind"] == "mixed" and case["coupling"] == "pc2":
        # (the half-step register of a particle that crossed a face: either image)
        out["x1"] = None
    return out


def _exact_output(p, S, x, v, m, blk, mom):
    p.place(x)
    d = m / S.vol
    f = p.deposit([d, d * v[0], d * v[1], d * v[2]])
    rho = f[0]
    acc = p.gather(mom)
    best = int(rho.reshape(-1).argmax())
    N1, N2, _ = S.N
    c = (best % N1, (best // N1) % N2, best // (N1 * N2))
    row = torch.tensor([float(m.numel()), float(m.sum())] + [float((m * v[a]).sum()) for a in range(3)]
                       + [float((0.5 * m * (v * v).sum(0)).sum()),
                          math.sqrt(float((m * x[2] ** 2).sum() / m.sum())), float(rho.max())]
                       + [S.lo[a] + (c[a] + 0.5) * S.dx for a in range(3)]
                       + [0.0, -1.0, -1.0, 0.0, 0.0], dtype=torch.float64, device=x.device)
    return {"x": x, "v": v, "block": blk.int(), "row": row, "science": _to_blocks(S, f),
            "density": _to_blocks(S, rho[None]), "acc": torch.stack(acc)}


def _exact_ensemble(case, seed):
    n = case["side"]
    dx, v0 = 1.0 / n, 0.1
    dt = 0.3 * dx / (1.0 + v0)
    f64 = dict(device="cuda", dtype=torch.float64)
    c = torch.arange(n ** 3, device="cuda")
    ctr = torch.stack([((c % n).double() + 0.5) * dx, (((c // n) % n).double() + 0.5) * dx,
                       ((c // n ** 2).double() + 0.5) * dx])
    outs = []
    for k, (taus, eps) in enumerate(_boxes(case, seed)):
        per = n ** 3 * case["ppc"]
        x = ctr.repeat(1, case["ppc"] * len(taus))
        ts = torch.tensor(taus, **f64).repeat_interleave(per)
        m = torch.tensor([e / per for e in eps], **f64).repeat_interleave(per)
        v = torch.zeros_like(x)
        v[0] = v0
        p = Plain((n, n, n), dx, [0.0] * 3, [1.0] * 3, 2, 2, True, x, v, ts, m,
                  torch.zeros((3, n, n, n), **f64))
        for _ in range(1 + case["cycles"]):
            p.imex(dt)
        outs.append(p)
    cat = lambda f: torch.cat([f(p) for p in outs], dim=1)           # noqa: E731
    per = n ** 3 * case["ppc"] * case["nspec"]
    return {"x": cat(lambda p: p.x), "v": cat(lambda p: p.v), "x1": cat(lambda p: p.x1),
            "v1": cat(lambda p: p.v1), "rate": cat(lambda p: p.R),
            "block": torch.arange(len(outs), device="cuda").repeat_interleave(per).int(),
            "gas": torch.stack([torch.cat([p.rho[None], p.mom]) for p in outs])}
