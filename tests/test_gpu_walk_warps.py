"""The group walk's two forms, one warp or four for a group, at the line between them (32,768 particles) and at the
edges of groups, leaves and chunks.

Neighbour sets exactly against the oracle's brute force. Gravity with θ → 0 and no local expansion is the direct sum in
f32 (terms good to a few 2^-24, at most 32,769 of them): 1e-5 RMS against FP64. (With the expansion it is not: a leaf of
one particle has no extent, is accepted at any θ and expanded where it is far.) Zero softening takes the loop that leaves a particle's own
term out by index."""
import math

import numpy as np
import pytest

import oracle
from botheadstudios_b200 import materials as M
from botheadstudios_b200.gpusph import GpuSph, particles_from_arrays

pytestmark = pytest.mark.gpu
LINE = 32_768


def _cloud(n, seed, h):
    rng = np.random.default_rng(seed)
    side = n ** (1.0 / 3.0)
    pos = rng.uniform(0.0, side, (n, 3)).astype(np.float32)
    return particles_from_arrays(pos, np.full(n, h) * rng.uniform(0.8, 1.2, n), np.zeros((n, 3)), np.full(n, 1e3),
                                 rng.uniform(0.5, 1.5, n), np.zeros(n, np.uint32))


def _check(p, K, quad, soft, theta=1.0e-4, local=0.0, bound=1.0e-5):
    n = len(p)
    with GpuSph(n, G=1.0, theta=theta, leaf_size=K, multipole=quad, max_neighbours=256, local_theta=local) as s:
        s.upload(p, M.eos_table(), soft)
        s.eval_forces()
        assert s.diag()["overflow_flags"] == 0
        nb, g = s.neighbour_sets(), s.inspect("ACC_GRAV")
    want = oracle.neighbours32(np.concatenate([p["pos"], p["h"][:, None]], 1), cap=256)
    assert all(np.array_equal(nb[i], want[i]) for i in range(n))
    tg = np.random.default_rng(1).choice(n, min(n, 1024), replace=False).astype(np.uint32)
    ref = oracle.gravity_direct64(p["pos"].astype(np.float64), p["mass"].astype(np.float64), soft, 1.0, targets=tg)
    err = math.sqrt(((g[tg, :3] - ref) ** 2).sum() / max((ref**2).sum(), 1e-300))
    assert np.isfinite(g).all() and err < bound, err


@pytest.mark.parametrize("n", [1, 31, 32, 33, 65, 1000])
@pytest.mark.parametrize("K,quad", [(1, 0), (8, 1), (16, 1), (32, 1)])
@pytest.mark.parametrize("soft", [0.0, 0.1])
def test_small_impacts(n, K, quad, soft):
    _check(_cloud(n, n + K, 2.2), K, quad, soft)


@pytest.mark.parametrize("n", [LINE, LINE + 1])
@pytest.mark.parametrize("soft", [0.0, 0.1])
def test_both_sides_of_the_line(n, soft):
    _check(_cloud(n, 7, 2.2), 16, 1, soft)
    _check(_cloud(n, 8, 2.2), 16, 1, soft, theta=0.6, local=0.3, bound=5e-3)  # the truncation of an opening angle of 0.6


def test_a_batch_across_the_line_equals_each_impact_alone():
    sizes = [LINE + 100, 12, LINE, 700]
    parts = [_cloud(n, 20 + n, 2.2) for n in sizes]
    off = np.concatenate([[0], np.cumsum(sizes)])
    kw = dict(G=1.0, theta=0.6, leaf_size=16, multipole=1, max_neighbours=256, kernel="wendland", h_mode=1,
              h_neighbours=32.0, h_iters=2)

    def run(p, offsets):
        with GpuSph(len(p), **kw) as s:
            s.upload_batch(p, offsets, M.eos_table(), 0.1)
            s.set_dt(1e-3)
            s.encode_kdk(2)
            d = s.diag()
            return s.readback(), s.inspect("ACC_GRAV"), d

    state, grav, d = run(np.concatenate(parts), off)
    assert d["overflow_flags"] == 0
    for k, p in enumerate(parts):
        one, g1, _ = run(p, [0, len(p)])
        a, b = off[k], off[k + 1]
        for f in ("pos", "vel", "h", "u", "rho"):
            assert np.array_equal(state[f][a:b], one[f]), (k, f)
        assert np.array_equal(grav[a:b], g1)


@pytest.mark.parametrize("n", [33, 1000, LINE + 1])
def test_heavy_particles_with_a_small_softening(n):
    """G m / soft³ beyond the f32 range: a particle's own (zero) force must not come out as infinity times zero."""
    p = _cloud(n, 5, 2.2)
    p["mass"] *= np.float32(1e30)
    for soft in (1e-2, 1e-3, 1e-4):
        _check(p, 16, 0, soft)


@pytest.mark.parametrize("K", [1, 2, 3, 5, 7, 11, 12, 16, 17, 24, 31, 32])
@pytest.mark.parametrize("n", [1, 100, 2000, LINE + 1])
def test_neighbours_of_the_per_particle_mode_in_leaves_of_any_size(K, n):
    p = _cloud(n, n + K, 2.2)
    with GpuSph(n, G=1.0, leaf_size=K, mac=1, max_neighbours=256) as s:
        s.upload(p, M.eos_table(), 0.1)
        s.eval_forces()
        assert s.diag()["overflow_flags"] == 0
        nb = s.neighbour_sets()
    want = oracle.neighbours32(np.concatenate([p["pos"], p["h"][:, None]], 1), cap=256)
    assert all(np.array_equal(nb[i], want[i]) for i in range(n))
