"""The work that users of this framework have it do, as timed cases over the real range of sizes.

A simulation run is: relax a body, assemble it into an impact, upload it, advance it step by step (one impact,
or many in one context) with the particle buffer handed to the renderer each frame, and measure the disk at the
end. Around that run there are the point-set gravity of a frame loop that may not allocate, the grain scene of
the ground view, and the training of the smoothing-length network. Every kind of case goes through the entry
points that such a program calls, in the configurations of botheadstudios_b200/workloads.py.

Inputs come from the framework's own seeded initial conditions (botheadstudios_b200/ic.py), so they hold what the
solver meets: two differentiated bodies on a collision course, planets, post-impact fields, packs of grains.
`exact` restates each path in plain torch in 64 bits: direct sums over all pairs for gravity, every pair inside
the support for the smoothed sums.
"""
import math

import numpy as np
import torch

from botheadstudios_b200 import _lib, grains, ic, learned_h, workloads
from botheadstudios_b200.gpusph import GpuSph

# The reference's plain method: cubic spline, fixed smoothing lengths, one particle per leaf, monopoles.
PLAIN = dict(kernel="cubic", theta=0.5, quad=0, leaf=1, h_mode=0, n_ngb=48.0, max_nbr=256)
# The method of the large impacts: Wendland C2, solved smoothing lengths, quadrupoles.
METHOD = dict(kernel="wendland", theta=0.6, quad=1, leaf=16, h_mode=1, n_ngb=64.0, max_nbr=192)

# A cautious Courant factor: a step costs the same, and the thousands of passes of a measurement stay in the
# approach and the first contact of the bodies, so that every pass meets the same distribution.
CFL = 0.02

GRAIN_PARAMS = dict(dt=2.0e-3, stiffness=4000.0, normal_damp=30.0, friction=0.6, tangent_damp=40.0, cohesion=5.0)
GRAIN_GROUND = dict(air_rho=1.2, drag_cd=0.5, specific_heat=800.0, cool_rate=0.05)
POINT_THETA = 0.5
RELAX_DAMP, RELAX_OMEGA = 0.98, 0.3
TRAIN_BATCH, TRAIN_LR = 4096, 2.0e-3


def listed():
    return [
        # the interactive scene: the small plain-method impact, a few substeps for each rendered frame
        dict(name="impact_10k", kind="step", n=10_240, substeps=4, graph=0, **PLAIN),
        # a survey run: the large impacts' method at low resolution, steady steps replayed from a graph
        dict(name="impact_65k", kind="step", n=65_536, substeps=2, graph=1, **METHOD),
        # the production impact
        dict(name="impact_1m", kind="step", n=1_048_576, substeps=1, graph=0, **METHOD),
        # the largest single impact
        dict(name="impact_4m", kind="step", n=4_194_304, substeps=1, graph=0, **METHOD),
        # a parameter sweep: 16 impacts of uneven size in one context
        dict(name="batch_16", kind="batch", impacts=16, n_min=20_000, n_max=200_000, substeps=2, graph=1, **METHOD),
        # an impact with the learned smoothing lengths, at an odd size
        dict(name="learned_300k", kind="step", n=299_993, substeps=1, graph=0, **dict(METHOD, h_mode=2)),
        # the relaxation of a spinning body before it is placed
        dict(name="relax_131k", kind="relax", n=131_072, substeps=2, **METHOD),
        # a host that keeps the state itself: upload, one step, readback
        dict(name="roundtrip_262k", kind="roundtrip", n=262_144, substeps=1, graph=0, **METHOD),
        # gravity of a point set inside a frame loop that may not allocate
        dict(name="points_16k", kind="points", n=16_001, leaf=16, quad=1),
        # the measurement that ends a run
        dict(name="measure_1m", kind="measure", n=1_000_000, ring=20_000, variant=0),
        # the ground scene: a pile of grains on terrain
        dict(name="grains_60k", kind="grains", n=60_000, substeps=4, terrain=96),
        # an epoch of the smoothing-length network's training (forward, backward, optimizer)
        dict(name="train_100k", kind="train", n=100_000),
    ]


def _spread(rng, lo, hi):
    """A size between lo and hi, even over its logarithm, as odd as it comes."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "step", "step", "batch", "learned", "relax", "roundtrip", "points", "measure",
                       "grains", "train"])
    if kind == "plain":
        return dict(kind="step", n=_spread(rng, 1_000, 50_000), substeps=rng.randint(1, 6), graph=rng.choice([0, 1]),
                    **PLAIN)
    method = dict(METHOD, leaf=rng.choice([8, 16, 16, 32]))
    if kind == "step":
        n = _spread(rng, 10_000, 3_000_000)
        return dict(kind="step", n=n, substeps=1 if n > 200_000 else rng.randint(1, 4), graph=rng.choice([0, 1]),
                    **method)
    if kind == "learned":
        return dict(kind="step", n=_spread(rng, 30_000, 1_500_000), substeps=1, graph=0, **dict(method, h_mode=2))
    if kind == "batch":
        low = _spread(rng, 5_000, 30_000)
        return dict(kind="batch", impacts=rng.randint(2, 24), n_min=low, n_max=low * rng.randint(2, 8),
                    substeps=rng.choice([1, 2]), graph=rng.choice([0, 1]), **method)
    if kind == "relax":
        return dict(kind="relax", n=_spread(rng, 10_000, 1_000_000), substeps=rng.randint(1, 2), **method)
    if kind == "roundtrip":
        return dict(kind="roundtrip", n=_spread(rng, 20_000, 2_000_000), substeps=rng.randint(1, 2), graph=0,
                    **method)
    if kind == "points":
        return dict(kind="points", n=_spread(rng, 1_000, 65_536), leaf=rng.choice([8, 16, 32]),
                    quad=rng.choice([0, 1]))
    if kind == "measure":
        n = _spread(rng, 60_000, 3_000_000)
        return dict(kind="measure", n=n, ring=max(2_000, n // rng.randint(40, 80)), variant=rng.choice([0, 1]))
    if kind == "grains":
        n = _spread(rng, 2_000, 300_000)
        return dict(kind="grains", n=n, substeps=rng.randint(1, 8), terrain=rng.choice([0, 64, 128]))
    return dict(kind="train", n=_spread(rng, 20_000, 400_000))


# ---- inputs and contexts ------------------------------------------------------------------------------------
def _bodies(case, seed):
    """The initial conditions of a case (host arrays, code units)."""
    kind = case["kind"]
    if kind == "batch":
        return _batch(case, seed)
    if kind == "relax":
        return ic.planet(case["n"], n_ngb=case["n_ngb"], seed=seed)
    small = case["n"] // 11
    return ic.impact(case["n"] - small, small, n_ngb=case.get("n_ngb", 64.0), seed=seed)


def _batch(case, seed):
    """Impacts of uneven size as ic.batch draws them; the seed changes the bodies and not the sizes."""
    parts, soft = [], []
    for d in _batch_draws(case):
        small = max(1, int(round(d["n"] * d["mass_ratio"] / (1.0 + d["mass_ratio"]))))
        b = ic.impact(d["n"] - small, small, n_ngb=case["n_ngb"], mass_ratio=d["mass_ratio"],
                      v_factor=d["v_factor"], angle_deg=d["angle_deg"], seed=d["seed"] + seed)
        parts.append(b.particles)
        soft.append(b.softening)
    offsets = np.concatenate([[0], np.cumsum([len(p) for p in parts])]).astype(np.uint32)
    return ic.Batch(particles=np.concatenate(parts), offsets=offsets, softening=np.asarray(soft, np.float32),
                    eos=b.eos, units=b.units, params=[])


def _batch_draws(case):
    return ic.batch_draws(case["impacts"], case["n_min"], case["n_max"], seed=case["impacts"])


def _solver_config(case, units, **over):
    return dict(theta=case["theta"], leaf_size=case["leaf"], kernel=case["kernel"], multipole=case["quad"],
                h_mode=case["h_mode"], h_neighbours=case["n_ngb"], h_iters=2, max_neighbours=case["max_nbr"],
                graph=case.get("graph", 0), **dict(dict(cfl=CFL), **over), **ic.config_kwargs(units))


def _relax_dt(bodies):
    """A relaxation step well inside the Courant limit of the coldest initial state (sound speeds are about 1)."""
    return 0.05 * float(bodies.particles["h"].min())


class _Memory:
    """The solver's buffer of n 48-byte particle records, for torch.as_tensor; it keeps the solver alive."""

    def __init__(self, solver, n):
        self.solver, address = solver, solver.particle_buffer()
        self.__cuda_array_interface__ = dict(shape=(n, 12), typestr="<f4", data=(address, False), version=3)


def _record_views(record):
    """The floating fields of 48-byte records seen as [n, 12] float32."""
    return dict(pos=record[:, 0:3], h=record[:, 3], vel=record[:, 4:7], u=record[:, 7], rho=record[:, 10])


def _pinned(n):
    """n particle records in pinned host memory, and the tensor that holds them."""
    t = torch.empty(n * 48, dtype=torch.uint8, pin_memory=True)
    return t.numpy().view(_lib.PARTICLE_DTYPE), t


def _terrain(size, seed):
    rng = np.random.default_rng(seed)
    a, b = rng.uniform(0.0, 2.0 * math.pi, 2)
    z, x = np.meshgrid(np.arange(size), np.arange(size), indexing="ij")
    return np.round(2.0 * np.sin(0.15 * x + a) + 2.0 * np.cos(0.11 * z + b)).astype(np.int32)


def _grain_pile(case, seed):
    """A dense pack of grains of half a metre on the terrain (or in free space), and the terrain's heights."""
    pile = grains.grain_pack(case["n"], seed=seed)
    pile["offset"] -= pile["offset"].mean(0)
    pile["u"] = 800.0 * np.random.default_rng(seed + 1).uniform(300.0, 1500.0, case["n"])
    heights = _terrain(case["terrain"], seed) if case["terrain"] else None
    if heights is not None:
        pile["offset"][:, 1] += heights.max() - 0.01 - pile["offset"][:, 1].min()
    return pile, heights


def _training_set(case, seed):
    """Rows of the network's eight features with the spreads that trajectories have, their targets, and a fresh
    network normalised to them."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    x = rng.normal(0.0, [5e-3, 0.15, 4e-3, 0.06, 0.3, 1.0, 0.1, 1.0], (n, 8))
    x[:, 5] = rng.random(n) < 0.3
    x[:, 6] = np.abs(x[:, 6])
    x[:, 7] = rng.random(n)
    t = 0.4 * x[:, 0] + x[:, 2] / 3.0 + 0.01 * np.sin(6.0 * x[:, 1]) * x[:, 4] + rng.normal(0.0, 2e-4, n)
    x, t = x.astype(np.float32), t.astype(np.float32)
    return learned_h.init_params(*learned_h.normalisation(x, t), seed=seed), x, t


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "batch", "relax"):
        b = _bodies(case, seed)
        s = GpuSph(len(b.particles), **_solver_config(case, b.units, **(dict(cfl=0.0) if kind == "relax" else {})))
        if case["h_mode"] == 2:
            s.mlp_set(learned_h.load())
            s.set_progress(0.5)
        if kind == "relax":
            s.set_dt(_relax_dt(b), RELAX_DAMP)
            s.set_av(0.0, 0.0)
            s.set_omega(RELAX_OMEGA)
        workloads.upload(s, b)
        record = torch.as_tensor(_Memory(s, len(b.particles)), device="cuda")
        return dict(kind=kind, solver=s, substeps=case["substeps"], out=_record_views(record))
    if kind == "roundtrip":
        b = _bodies(case, seed)
        s = GpuSph(len(b.particles), **_solver_config(case, b.units))
        sent, keep_sent = _pinned(len(b.particles))
        back, keep_back = _pinned(len(b.particles))
        sent[:] = b.particles
        out = _record_views(back.view(np.float32).reshape(-1, 12))
        return dict(kind=kind, solver=s, substeps=case["substeps"], sent=sent, back=back, eos=b.eos,
                    softening=b.softening, out=out, keep=(keep_sent, keep_back))
    if kind == "points":
        b = _bodies(case, seed)
        body = torch.as_tensor(np.concatenate([b.particles["pos"], b.particles["mass"][:, None]], 1), device="cuda")
        acc = torch.empty_like(body)
        return dict(kind=kind, call=_lib.load().sph_gravity_tree_noalloc, n=case["n"], leaf=case["leaf"],
                    quad=case["quad"], body=body, acc=acc, softening=b.softening)
    if kind == "measure":
        p = ic.post_impact_scene(**_field(case), seed=seed)
        s = GpuSph(len(p), leaf_size=16, max_neighbours=8)  # the field is measured, not advanced
        s.upload(p, ic.eos_table(), 0.0)
        return dict(kind=kind, solver=s, variant=case["variant"])
    if kind == "grains":
        pile, heights = _grain_pile(case, seed)
        s = grains.GpuGrains(case["n"])
        s.set_params(**GRAIN_PARAMS)
        s.set_ground(center=(0.5 * case["terrain"], 0.0, 0.5 * case["terrain"]), **GRAIN_GROUND)
        s.set_terrain(heights)
        s.replace(pile)
        return dict(kind=kind, scene=s, substeps=case["substeps"])
    params, x, t = _training_set(case, seed)
    return dict(kind=kind, params=params, x=x, t=t, seed=seed)


def _field(case):
    """A post-impact field of n remnant particles, scaled as workloads.MEASURE_WORKLOADS scales it."""
    one = workloads.MEASURE_WORKLOADS["post_impact_1m"]
    f = (1.0e6 / case["n"]) ** (1.0 / 3.0)
    return dict(n_rem=case["n"], n_ring=case["ring"], n_esc=max(100, case["n"] // 500), clumps=one["clumps"],
                m_rem=6.0e24 / case["n"], h_rem=2.5e5 * f, h_debris=1.2e5, clump_radius=4.0e5)


MEASURED = ("earth_frac", "disk_mass", "disk_target", "disk_impactor", "remnant_target", "remnant_impactor",
            "escaped_target", "escaped_impactor", "r_remnant", "m_remnant", "clump_mass", "clump_target_frac")
COUNTED = ("clump_n", "n_clumps", "n_bound", "n_disk")


def run(state):
    kind = state["kind"]
    if kind in ("step", "batch", "relax"):
        s = state["solver"]
        if kind == "relax":
            s.encode_relax(state["substeps"])
        else:
            s.encode_kdk(state["substeps"])
        s.particle_buffer()
        return state["out"]
    if kind == "roundtrip":
        s = state["solver"]
        s.upload(state["sent"], state["eos"], state["softening"])
        s.encode_kdk(state["substeps"])
        s.readback_into(state["back"])
        return state["out"]
    if kind == "points":
        st = state["call"](state["body"].data_ptr(), state["n"], 1.0, state["softening"], POINT_THETA, state["leaf"],
                           state["quad"], state["acc"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if st != _lib.SPH_OK:
            raise RuntimeError(f"sph_gravity_tree_noalloc: status {st}")
        return dict(acc=state["acc"][:, :3], phi=state["acc"][:, 3])
    if kind == "measure":
        m = state["solver"].measure_disk(variant=state["variant"])
        return dict(values=np.array([m[k] for k in MEASURED]), counts=np.array([m[k] for k in COUNTED], np.int64))
    if kind == "grains":
        state["scene"].dispatch(state["substeps"])
        g = state["scene"].readback()
        return dict(offset=g["offset"], vel=g["vel"], u=g["u"], resting=g["resting"])
    params, losses = learned_h.train(state["params"], state["x"], state["t"], epochs=1, batch=TRAIN_BATCH,
                                     lr=TRAIN_LR, seed=state["seed"])
    return dict(params=params, losses=losses)


def work(case):
    kind = case["kind"]
    if kind == "train":
        return dict(bytes=36.0 * case["n"], flops=3.0 * 2.0 * (8 * 64 + 64 * 64 + 64) * case["n"])
    if kind == "measure":
        # two readings of 40 bytes (the remnant's radius has to be known before the orbits), ~100 operations each
        return dict(bytes=80.0 * (case["n"] + case["ring"]), flops=100.0 * (case["n"] + case["ring"]))
    if kind == "grains":
        # the records and about eight contacts of a grain, ~90 operations each; the records go to the host once
        return dict(bytes=case["n"] * (80.0 + 128.0 * case["substeps"]), flops=case["n"] * 900.0 * case["substeps"])
    if kind == "points":
        return dict(bytes=32.0 * case["n"], flops=_tree_flops(case["n"], POINT_THETA, case["quad"]) * case["n"])
    if kind == "batch":
        n = sum(d["n"] for d in _batch_draws(case))
    else:
        n = case["n"]
    # state read and written once a substep; the tree's interactions, and the smoothed sums over half the target
    # count of pairs: forces twice, density once for each pass of the solve
    passes = 3.0 if case["h_mode"] else 1.0
    pairs = case["n_ngb"] * (30.0 * passes + 60.0 * (1.0 if kind == "relax" else 2.0))
    flops = case["substeps"] * n * (_tree_flops(n, case["theta"], case["quad"]) + pairs)
    link = 96.0 * n if kind == "roundtrip" else 48.0 * n
    return dict(bytes=link + 136.0 * n * case["substeps"], flops=flops)


def _tree_flops(n, theta, quad):
    """Operations for one particle of a Barnes-Hut sum over n: about 28 theta^-3 accepted nodes in each of the
    levels of an eightfold tree, 20 operations for a monopole and 65 for a quadrupole."""
    return 28.0 / theta**3 * max(1.0, math.log(n, 8) - 1.0) * (65.0 if quad else 20.0)


# ---- the same in 64 bits ------------------------------------------------------------------------------------
DIRECT_PAIRS = 2.5e11  # pairs of direct sums in one answer, about ten seconds


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "measure":
        return _exact_measure(case, seed)
    if kind == "grains":
        return _exact_grains(case, seed)
    b = _bodies(case, seed)
    n = len(b.particles)
    if kind == "points":
        p = _cuda(b.particles["pos"])
        m = _cuda(b.particles["mass"])
        acc, phi = _gravity(p, m, float(np.float32(b.softening)) ** 2, 1.0)
        return dict(acc=acc, phi=phi)
    evals = case["substeps"] + (0 if kind == "relax" else 1)
    offsets = b.offsets if kind == "batch" else np.array([0, n])
    if case["h_mode"] == 2 or evals * float((np.diff(offsets).astype(np.float64) ** 2).sum()) > DIRECT_PAIRS:
        return None  # which proposals are accepted is a decision; and the direct sum of a large body takes too long
    parts = []
    for k in range(len(offsets) - 1):
        soft = b.softening[k] if kind == "batch" else b.softening
        body = _Body(case, b, b.particles[offsets[k]:offsets[k + 1]], float(np.float32(soft)))
        parts.append(body.relax(case["substeps"], _relax_dt(b)) if kind == "relax" else body.advance(case["substeps"]))
    return {f: torch.cat([p[f] for p in parts]) for f in parts[0]}


def _cuda(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda").double()


def _gravity(pos, mass, soft2, G):
    """Direct softened sum over all pairs: accelerations and potentials."""
    n = len(mass)
    rows = max(1, int(3.0e7) // n)
    acc, phi = torch.empty_like(pos), torch.empty_like(mass)
    for a in range(0, n, rows):
        d = [pos[:, k] - pos[a:a + rows, k, None] for k in range(3)]
        inv = (d[0] * d[0]).addcmul_(d[1], d[1]).addcmul_(d[2], d[2]).add_(soft2).rsqrt_()
        me = torch.arange(a, min(a + rows, n), device=pos.device)
        inv[me - a, me] = 0.0
        phi[a:a + rows] = -G * (inv @ mass)
        w = inv.pow_(3).mul_(mass)
        for k in range(3):
            acc[a:a + rows, k] = G * (w * d[k]).sum(1)
    return acc, phi


def _near_pairs(pos, reach):
    """All ordered pairs i != j closer than (reach_i + reach_j)/2, from a grid of cells of the largest reach."""
    cell = torch.floor((pos - pos.min(0).values) / (reach.max() * 1.0001)).long() + 1
    size = cell.max(0).values + 2
    key = (cell[:, 0] * size[1] + cell[:, 1]) * size[2] + cell[:, 2]
    order = torch.argsort(key)
    skey = key[order].contiguous()
    first, second = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                want = key + (dx * size[1] + dy) * size[2] + dz
                lo, hi = torch.searchsorted(skey, want), torch.searchsorted(skey, want, right=True)
                count = hi - lo
                i = torch.repeat_interleave(torch.arange(len(key), device=pos.device), count)
                start = torch.cumsum(count, 0) - count
                j = order[lo[i] + torch.arange(len(i), device=pos.device) - start[i]]
                d = pos[i] - pos[j]
                keep = ((d * d).sum(1) < (0.5 * (reach[i] + reach[j])) ** 2) & (i != j)
                first.append(i[keep])
                second.append(j[keep])
    return torch.cat(first), torch.cat(second)


class _Body:
    """One impact (or planet) advanced in 64 bits with the solver's method."""

    def __init__(self, case, bodies, p, softening):
        self.pos, self.h, self.vel = _cuda(p["pos"]), _cuda(p["h"]), _cuda(p["vel"])
        self.u, self.mass = _cuda(p["u"]), _cuda(p["mass"])
        self.eos = _cuda(bodies.eos)[torch.as_tensor(p["mat"].astype(np.int64), device="cuda")].T
        self.units, self.soft2 = bodies.units, softening * softening
        self.wendland, self.solve = case["kernel"] == "wendland", case["h_mode"] == 1
        self.eta = ic.eta_for(case["n_ngb"])
        self.alpha, self.beta = 1.0, 2.0
        self.skin, self.tol, self.iters = 0.15, 1.0e-3, 2

    def kernel(self, r, h):
        """W, dW/dr and dW/dh of the pair kernels with support h."""
        q = r / h
        t = (1.0 - q).clamp(min=0.0)
        if self.wendland:
            c, f, fp = 21.0 / (2.0 * math.pi), t**4 * (1.0 + 4.0 * q), -20.0 * q * t**3
        else:
            s = (0.5 - q).clamp(min=0.0)
            c, f, fp = 8.0 / math.pi, 2.0 * t**3 - 8.0 * s**3, 24.0 * s**2 - 6.0 * t**2
        return c / h**3 * f, c / h**4 * fp, -c / h**4 * (3.0 * f + q * fp)

    def density(self):
        i, j, r = self.i, self.j, self.r
        hij = 0.5 * (self.h[i] + self.h[j])
        w, _, dwdh = self.kernel(r, hij)
        w0, _, dw0 = self.kernel(torch.zeros_like(self.h), self.h)
        rho = (self.mass * w0).index_add_(0, i, self.mass[j] * w)
        drho = (self.mass * dw0).index_add_(0, i, 0.5 * self.mass[j] * dwdh)
        return rho, drho

    def rebuild(self):
        grown = self.h * (1.0 + self.skin if self.solve else 1.0)
        self.i, self.j = _near_pairs(self.pos, grown)
        self.d = self.pos[self.i] - self.pos[self.j]
        self.r = (self.d * self.d).sum(1).sqrt()
        h0 = self.h.clone()
        if self.solve:
            for _ in range(self.iters):
                rho, drho = self.density()
                rt = self.mass * self.eta**3 / self.h**3
                step = -(rho - rt) / (drho + 3.0 * rt / self.h)
                h = torch.minimum(torch.maximum(self.h + step, 0.8 * self.h), 1.2 * self.h)
                h = torch.minimum(h, h0 * (1.0 + self.skin) * 0.999)
                self.h = torch.maximum(h, h0 / ((1.0 + self.skin) * 1.001))
        self.rho, _ = self.density()
        if self.solve:
            res = ((self.rho - self.mass * self.eta**3 / self.h**3) / self.rho).abs().max()
            self.skin = 0.15 if res > 10.0 * self.tol else 0.05
        self.grav, _ = _gravity(self.pos, self.mass, self.soft2, self.units.G)

    def pressure(self, rho, u):
        rho0, a, b, A, B, e0, e_iv, e_cv, al, be = self.eos[:10]
        r = rho.clamp(min=self.units.rho_floor)
        eta = r / rho0
        mu, omega = eta - 1.0, u / (e0 * eta * eta) + 1.0
        cold = (a + b / omega) * r * u + A * mu + B * mu * mu
        z = rho0 / r - 1.0
        hot = a * r * u + (b * r * u / omega + A * mu * torch.exp(-be * z)) * torch.exp(-al * z * z)
        mixed = ((u - e_iv) * hot + (e_cv - u) * cold) / (e_cv - e_iv)
        return torch.where((eta >= 1.0) | (u <= e_iv), cold, torch.where(u >= e_cv, hot, mixed))

    def forces(self):
        rho, u, i, j = self.rho, self.u, self.i, self.j
        p = self.pressure(rho, u)
        dr, du = rho * 1.0e-3, u.abs() * 1.0e-3 + self.units.du_floor
        dpdr = (self.pressure(rho + dr, u) - self.pressure(rho - dr, u)) / (2.0 * dr)
        dpdu = (self.pressure(rho, u + du) - self.pressure(rho, u - du)) / (2.0 * du)
        c = (dpdr + p / rho**2 * dpdu).clamp(min=0.0).sqrt()
        hij = 0.5 * (self.h[i] + self.h[j])
        _, dw, _ = self.kernel(self.r, hij)
        v = self.vel[i] - self.vel[j]
        vr = (v * self.d).sum(1)
        mu = hij * vr.clamp(max=0.0) / (self.r**2 + 0.01 * hij**2)
        visc = (self.beta * mu - self.alpha * 0.5 * (c[i] + c[j])) * mu / (0.5 * (rho[i] + rho[j]))
        pr = p / rho**2
        s = (pr[i] + pr[j] + visc) * self.mass[j] * torch.where(self.r > self.units.r_min, dw / self.r, 0.0 * dw)
        acc = self.grav.index_add(0, i, -s[:, None] * self.d)
        heat = torch.zeros_like(u).index_add_(0, i, 0.5 * s * vr)
        signal = (self.h / (c + self.vel.norm(dim=1)).clamp(min=self.units.sig_floor)).min()
        return acc, heat, signal

    def kick(self, acc, heat, half):
        self.vel = self.vel + acc * half
        self.u = (self.u + heat * half).clamp(min=0.0)

    def result(self):
        return dict(pos=self.pos, h=self.h, vel=self.vel, u=self.u, rho=self.rho)

    def advance(self, substeps):
        self.rebuild()
        for _ in range(substeps):
            acc, heat, signal = self.forces()
            dt = CFL * signal
            self.kick(acc, heat, 0.5 * dt)
            self.pos = self.pos + self.vel * dt
            self.rebuild()
            acc, heat, _ = self.forces()
            self.kick(acc, heat, 0.5 * dt)
        return self.result()

    def relax(self, steps, dt):
        self.alpha = self.beta = 0.0
        spin = torch.tensor([RELAX_OMEGA**2, RELAX_OMEGA**2, 0.0], device="cuda", dtype=torch.float64)
        for _ in range(steps):
            self.rebuild()
            acc, _, _ = self.forces()
            self.vel = (self.vel + (acc + spin * self.pos) * dt) * RELAX_DAMP
            self.pos = self.pos + self.vel * dt
        return self.result()


def _groups(n, i, j):
    """The connected components of n points with links (i, j): each point's smallest reachable index."""
    label = torch.arange(n, device=i.device)
    while True:
        low = label.scatter_reduce(0, i, label[j], "amin")
        low = low[low]
        if bool((low == label).all()):
            return label
        label = low


def _exact_measure(case, seed):
    p = ic.post_impact_scene(**_field(case), seed=seed)
    pos, vel, mass, h, rho = (_cuda(p[f]) for f in ("pos", "vel", "mass", "h", "rho"))
    target = torch.as_tensor(p["prov"].astype(np.int64), device="cuda") == 0
    G, M, m1 = _lib.default_config().G, mass.sum(), mass[:, None]
    com, vcom = (pos * m1).sum(0) / M, (vel * m1).sum(0) / M
    x, v = pos - com, vel - vcom
    r, order = x.norm(dim=1).sort(stable=True)
    cum = mass[order].cumsum(0)
    at = int(torch.searchsorted(cum, 0.85 * M).clamp(max=len(cum) - 1))
    r_rem, m_rem = r[at], cum[at]
    mu = G * m_rem
    r = x.norm(dim=1)
    energy = 0.5 * (v * v).sum(1) - mu / r
    ang2 = (torch.linalg.cross(x, v) ** 2).sum(1)
    peri = -mu / (2.0 * energy) * (1.0 - (1.0 + 2.0 * energy * ang2 / mu**2).clamp(min=0.0).sqrt())
    bound = energy < 0.0
    disk = bound & (peri > r_rem)
    kinds = [disk, bound & ~disk, ~bound]
    sums = [float(mass[k & t].sum()) for k in kinds for t in (target, ~target)]
    idx = disk.nonzero()[:, 0]
    link = 2.0 * (h[idx].mean() if case["variant"] == 0 else h.mean())
    # variant 0 measures links on single-precision differences, so candidates are taken a little further out
    q = pos[idx]
    i, j = _near_pairs(q, torch.full_like(h[idx], float(link) * 1.00001))
    d = q[i] - q[j]
    d = d.float().double() if case["variant"] == 0 else d
    keep = (d * d).sum(1) <= link * link
    label = _groups(len(idx), i[keep], j[keep])
    best, found, n_bound, n_groups = 0.0, (0.0, 0), 0, 0
    rho_rem = m_rem / (4.0 / 3.0 * math.pi * r_rem**3)
    values, members = label.unique(return_counts=True)
    for g in values[members > 1].tolist():
        k = idx[label == g]
        mk, n_groups = mass[k], n_groups + 1
        total = mk.sum()
        cv, cp = (vel[k] * mk[:, None]).sum(0) / total, (pos[k] * mk[:, None]).sum(0) / total
        kinetic = 0.5 * (mk * ((vel[k] - cv) ** 2).sum(1)).sum()
        volume = (mk / (rho[k] if case["variant"] == 0 else rho[k].clamp(min=1.0))).sum()
        potential = 0.0
        for a in range(0, len(k), 1024):
            d = pos[k][a:a + 1024, None, :] - pos[k][None, :, :]
            if case["variant"] == 0:
                dist = d.float().double().norm(dim=2).clamp(min=1.0)
            else:
                dist = ((d * d).sum(2) + 1.0e8).sqrt()
            inv = 1.0 / dist
            me = torch.arange(a, min(a + 1024, len(k)), device=d.device)
            inv[me - a, me] = 0.0
            potential -= 0.5 * G * float((mk[a:a + 1024, None] * inv * mk).sum())
        if float(kinetic) + potential < 0.0:
            n_bound += 1
            roche = 2.44 * r_rem * (rho_rem / (total / volume)) ** (1.0 / 3.0)
            if float((cp - com).norm()) > float(roche) and float(total) > best:
                best = float(total)
                found = (100.0 * float(mk[target[k]].sum()) / best, len(k))
    disk_mass = sums[0] + sums[1]
    values = [100.0 * sums[0] / disk_mass if disk_mass else 0.0, disk_mass, *sums, float(r_rem), float(m_rem), best,
              found[0]]
    return dict(values=np.array(values), counts=np.array([found[1], n_groups, n_bound, len(idx)], np.int64))


def _exact_grains(case, seed):
    """The contact law, the implicit velocity solve and the ground of the grain scene in 64 bits."""
    pile, heights = _grain_pile(case, seed)
    x, v, u, r, rho = (_cuda(pile[f]) for f in ("offset", "vel", "u", "radius", "rho"))
    dt, k, dn = (GRAIN_PARAMS[f] for f in ("dt", "stiffness", "normal_damp"))
    mu, dt_, coh = (GRAIN_PARAMS[f] for f in ("friction", "tangent_damp", "cohesion"))
    theta, reach, heat = 0.7, 0.15, GRAIN_GROUND["specific_heat"]
    field = None if heights is None else _cuda(heights)
    half = 0.5 * case["terrain"]

    def surface(px, pz):
        """Height and horizontal gradient of the bilinear surface under a position, and its normal."""
        ax, az = px + half, pz + half
        cx, cz = ax.floor(), az.floor()
        top = lambda a, b: field[b.clamp(0, len(field) - 1).long(), a.clamp(0, len(field) - 1).long()] - 0.5  # noqa: E731
        h00, h10, h01, h11 = top(cx, cz), top(cx + 1, cz), top(cx, cz + 1), top(cx + 1, cz + 1)
        fx, fz = ax - cx, az - cz
        gx = (h10 - h00) * (1 - fz) + (h11 - h01) * fz
        gz = (h01 - h00) * (1 - fx) + (h11 - h10) * fx
        height = (h00 * (1 - fx) + h10 * fx) * (1 - fz) + (h01 * (1 - fx) + h11 * fx) * fz
        normal = torch.stack([-gx, torch.ones_like(gx), -gz], 1)
        return height, normal / normal.norm(dim=1, keepdim=True)

    for _ in range(case["substeps"]):
        i, j = _near_pairs(x, 2.0 * r + reach)
        d = x[i] - x[j]
        dist = d.norm(dim=1)
        n = d / dist[:, None]
        overlap = r[i] + r[j] - dist
        w = v[i] - v[j]
        push = k * overlap.clamp(min=0.0)
        pull = coh * (1.0 - (-overlap).clamp(min=0.0) / reach).clamp(0.0, 1.0)
        wt = w - n * (w * n).sum(1, keepdim=True)
        slip = wt.norm(dim=1)
        drag = torch.minimum(torch.minimum(dt_ * slip, mu * (push + pull)), slip / dt)
        drag = torch.where(slip > 1e-9, drag / slip, 0.0 * slip)
        acc = torch.zeros_like(x).index_add_(0, i, n * (push - pull)[:, None] - wt * drag[:, None])
        g = torch.where(overlap > 0.0, theta * theta * dt * dt * k + theta * dt * dn, 0.0)
        nn = g[:, None, None] * n[:, :, None] * n[:, None, :]
        S = torch.zeros(len(x), 3, 3, device=x.device, dtype=x.dtype).index_add_(0, i, nn)
        coupling = torch.zeros_like(x).index_add_(0, i, (nn @ v[j][:, :, None])[:, :, 0])
        u = heat * 300.0 + (u - heat * 300.0) * math.exp(-GRAIN_GROUND["cool_rate"] * dt)
        speed = v.norm(dim=1, keepdim=True)
        air = 0.5 * GRAIN_GROUND["air_rho"] * GRAIN_GROUND["drag_cd"] * speed / (rho * 2.0 * r)[:, None]
        acc = acc - air * v + torch.tensor([0.0, -9.81, 0.0], device=x.device, dtype=x.dtype)
        rhs = v - (1.0 - theta) / theta * (S @ v[:, :, None])[:, :, 0] + coupling / theta + acc * dt
        new = torch.linalg.solve(torch.eye(3, device=x.device, dtype=x.dtype) + S, rhs)
        room = torch.full_like(r, 1.0e30)
        if field is not None:
            _, up = surface(x[:, 0], x[:, 2])
            gap = torch.where(((x[j] - x[i]) * up[i]).sum(1) > 0.0, (-overlap).clamp(min=0.0), 1.0e30)
            room = room.scatter_reduce(0, i, gap, "amin")
        x, v = x + 0.5 * dt * (v + new), new
        if field is not None:
            height, up = surface(x[:, 0], x[:, 2])
            depth = height - (x[:, 1] - r)
            hit = depth > 0.0
            stop = torch.where(hit, (-(v * up).sum(1)).clamp(min=0.0), 0.0)
            v = v + stop[:, None] * up
            t = v - (v * up).sum(1, keepdim=True) * up
            slip = t.norm(dim=1)
            lost = torch.where(hit & (slip > 1e-9), torch.minimum(mu * stop, slip) / slip.clamp(min=1e-9), 0.0)
            v = v - t * lost[:, None]
            lift = torch.minimum(depth.clamp(max=0.01), room)
            x = x + torch.where(hit, lift, 0.0)[:, None] * up
    return dict(offset=x, vel=v, u=u, resting=None)  # the settle counter counts threshold crossings


def _shuffled(n, seed):
    """The epoch's sample order: Fisher-Yates with the SplitMix64 sequence of the seed."""
    mask, order = (1 << 64) - 1, list(range(n))
    state = (seed * 0x2545F4914F6CDD1D + 1) & mask
    for i in range(n - 1, 0, -1):
        state = (state + 0x9E3779B97F4A7C15) & mask
        z = state
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (i + 1)
        order[i], order[j] = order[j], order[i]
    return order


def _exact_train(case, seed):
    params, x, t = _training_set(case, seed)
    p = _cuda(params)
    h = learned_h
    x = (_cuda(x) - p[h.XM:h.XM + 8]) * p[h.XS:h.XS + 8]
    t = (_cuda(t) - p[h.YM]) / p[h.YS]
    order = torch.as_tensor(_shuffled(case["n"], seed & 0xFFFFFFFF), device="cuda")
    w = p[:h.XM].clone()
    m1, m2, loss, step = torch.zeros_like(w), torch.zeros_like(w), 0.0, 0
    for a in range(0, case["n"], TRAIN_BATCH):
        pick = order[a:a + TRAIN_BATCH]
        w = w.detach().requires_grad_(True)
        a1 = torch.nn.functional.gelu(x[pick] @ w[h.W1:h.B1].view(8, 64) + w[h.B1:h.W2])
        a2 = torch.nn.functional.gelu(a1 @ w[h.W2:h.B2].view(64, 64) + w[h.B2:h.W3])
        err = a2 @ w[h.W3:h.B3] + w[h.B3] - t[pick]
        (err * err).mean().backward()
        loss, g, step = loss + float((err * err).sum()), w.grad, step + 1
        m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
        w = w.detach() - TRAIN_LR * (m1 / (1.0 - 0.9**step)) / ((m2 / (1.0 - 0.999**step)).sqrt() + 1.0e-8)
    return dict(params=torch.cat([w, p[h.XM:]]), losses=np.array([loss / case["n"]]))
