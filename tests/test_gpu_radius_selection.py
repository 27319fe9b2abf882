"""The remnant radius's selection at the sizes and distances where it can go wrong: one point, one past a block's stride,
a great many equal radii (ranked by further digits above 1,024), massless points, points far below the largest
coordinate (they share the first digit's last bin), mass fractions up to one.

Coordinates and masses are small integers, so the centre is exactly the origin and every running mass is exact: the
radius must be the f64 distance to within the three roundings of the sum of squares and its root, and the running mass
must be the very number."""
import math

import numpy as np
import pytest

import disk_scene as ds

CORNERS = np.array([[sx * a, sy * b, sz * c] for a, b, c in ((1, 2, 3), (2, 3, 1), (3, 1, 2))
                    for sx in (1, -1) for sy in (1, -1) for sz in (1, -1)], np.float32)


def _shells(n, distinct):
    """n points in antipodal pairs of equal mass on `distinct` shells."""
    k = np.arange(n // 2) % distinct
    half = CORNERS[(np.arange(n // 2) * 5) % len(CORNERS)] * (1.0 + k)[:, None].astype(np.float32)
    return np.concatenate([half, -half, np.zeros((n % 2, 3), np.float32)])


CASES = {
    "one": (np.zeros((1, 3), np.float32), None),
    "two": (_shells(2, 1), None),
    "odd": (_shells(257, 40), None),
    "one shell": (_shells(3000, 1), "index"),
    "two shells": (_shells(5001, 2), "index"),
    "many": (_shells(151_553, 900), None),
    "massless": (_shells(4000, 300), "every third"),
    "far point": (np.concatenate([_shells(2600, 700), [[2.0 ** 40, 0, 0]]]).astype(np.float32), "last massless"),
    "far below": (np.concatenate([_shells(2600, 700), [[2.0 ** 61, 0, 0]]]).astype(np.float32), "last massless"),
}


def _masses(pos, how):
    n = len(pos)
    m = np.full(n, 3.0, np.float32)
    pair = np.arange(n) % max(n // 2, 1)
    if how == "index":
        m = (1.0 + pair % 7).astype(np.float32)
    elif how == "every third":
        m[pair % 3 == 0] = 0.0
    elif how == "last massless":
        m[-1] = 0.0
    return m


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CASES))
def test_gpu_radius_crossing(name):
    from botheadstudios_b200 import ic, materials
    from botheadstudios_b200.gpusph import GpuSph
    pos, how = CASES[name]
    n = len(pos)
    p = np.zeros(n, ds.scene(0, n_rem=10, n_ring=0, n_esc=0, clumps=()).dtype)
    p["pos"], p["mass"], p["h"], p["rho"] = pos, _masses(pos, how), 1.0, 1.0
    assert not (pos.astype(np.float64) * p["mass"].astype(np.float64)[:, None]).sum(0).any() or n == 1
    rad = np.sqrt((pos.astype(np.float64) ** 2).sum(1))
    order = np.argsort(rad, kind="stable")
    cum = np.cumsum(p["mass"].astype(np.float64)[order])
    with GpuSph(n, **ic.config_kwargs(materials.SI)) as s:
        s.upload(p, ds.eos(), 1.0e4)
        for frac in (1e-9, 0.25, 0.5, 0.85, 1.0):
            k = int(np.argmax(cum >= frac * cum[-1]))
            got = s.measure_disk(0, remnant_frac=frac)
            assert got["m_remnant"] == cum[k], (frac, got["m_remnant"], cum[k])
            assert math.isclose(got["r_remnant"], rad[order][k], rel_tol=4 * 2.0 ** -53), frac


def _ball_bulk(pos, m):
    """body_bulk's last round in f64: every point stays in the clip sphere here (98 % of the mass of a shell or a lattice
    ball lie within 1.5 times its radius)."""
    rad = np.sqrt((pos.astype(np.float64) ** 2).sum(1))
    order = np.argsort(rad, kind="stable")
    cum = np.cumsum(m.astype(np.float64)[order])
    return rad[order][int(np.argmax(cum >= 0.98 * cum[-1]))]


MANY = {
    "1025 at one radius": lambda: _shells(1025, 1),
    "a shell in f32": lambda: _f32_shell(60_000),
    "half at one radius": lambda: np.concatenate([_shells(40_000, 1), _shells(40_000, 200)]),
    "a lattice ball": lambda: _lattice(45),
    "far below, one radius": lambda: np.concatenate([_shells(5000, 1), [[2.0 ** 61, 0, 0]]]).astype(np.float32),
}


def _f32_shell(n):
    v = np.random.default_rng(4).normal(size=(n // 2, 3))
    v = (v / np.linalg.norm(v, axis=1)[:, None]).astype(np.float32)
    return np.concatenate([v, -v])


def _lattice(r):
    k = np.arange(-r, r + 1)
    g = np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)
    return g[(g**2).sum(1) < r * r].astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(MANY))
def test_gpu_many_candidates(name):
    """More than 1,024 points share the crossing's first digits: the host asks for the others, in the remnant radius and
    in the bulk radius, and the call after it has few again."""
    from botheadstudios_b200 import ic, materials
    from botheadstudios_b200.gpusph import GpuSph
    pos = MANY[name]()
    n = len(pos)
    far = name.startswith("far")
    p = np.zeros(n, ds.scene(0, n_rem=10, n_ring=0, n_esc=0, clumps=()).dtype)
    p["pos"], p["mass"], p["h"], p["rho"] = pos, 3.0, 1.0, 1.0
    if far:
        p["mass"][-1] = 0.0
    rad = np.sqrt((pos.astype(np.float64) ** 2).sum(1))
    order = np.argsort(rad, kind="stable")
    cum = np.cumsum(p["mass"].astype(np.float64)[order])
    with GpuSph(n, **ic.config_kwargs(materials.SI)) as s:
        s.upload(p, ds.eos(), 1.0e4)
        for frac in (0.85, 1e-9, 0.3, 1.0):
            k = int(np.argmax(cum >= frac * cum[-1]))
            got = s.measure_disk(0, remnant_frac=frac)
            assert got["m_remnant"] == cum[k], (frac, got["m_remnant"], cum[k])
            assert math.isclose(got["r_remnant"], rad[order][k], rel_tol=4 * 2.0 ** -53), frac
        if not far:
            centre, mass, radius = s.body_bulk(0)
            assert not np.any(centre) and mass == cum[-1]
            assert math.isclose(radius, _ball_bulk(pos, p["mass"]), rel_tol=4 * 2.0 ** -53)
