"""The sort's bounded waits run out (a limit of no polls: every wait gives up at once, so the sort's result is no
permutation). A rebuild then goes on with the particles in the order they had, which any result that does not depend on
the order must not show; the measurement, which needs its order, fails; and both are right again with the next call.

Neighbour sets exactly against the oracle; gravity with an opening angle near zero is the direct sum in f32 (terms good to
a few 2^-24, at most 6,000 of them): 1e-5 RMS against FP64."""
import numpy as np
import pytest

import disk_scene as ds
import oracle
from botheadstudios_b200 import materials as M
from botheadstudios_b200.gpusph import GpuSph, SphError, particles_from_arrays

pytestmark = pytest.mark.gpu
SORT_TIMEOUT = 16
DEFAULT_POLLS = 1 << 21


def _polls(s, limit):
    assert s._L.sph_set_sort_polls(s._h, limit) == 0


def _cloud(n, seed):
    rng = np.random.default_rng(seed)
    return particles_from_arrays(rng.uniform(0.0, n ** (1.0 / 3.0), (n, 3)), rng.uniform(1.8, 2.6, n), np.zeros((n, 3)),
                                 np.full(n, 1e3), rng.uniform(0.5, 1.5, n), np.zeros(n, np.uint32))


def _rms(a, ref):
    return np.sqrt(((a - ref) ** 2).sum() / (ref**2).sum())


@pytest.mark.parametrize("mac", [0, 1])
@pytest.mark.parametrize("sizes", [[6000], [2500, 40, 3000]])
def test_a_rebuild_without_its_sort_gives_the_same_forces(mac, sizes):
    parts = [_cloud(n, n) for n in sizes]
    off = np.concatenate([[0], np.cumsum(sizes)])
    want = [oracle.neighbours32(np.concatenate([p["pos"], p["h"][:, None]], 1), cap=256) for p in parts]
    ref = [oracle.gravity_direct64(p["pos"].astype(np.float64), p["mass"].astype(np.float64), 0.1, 1.0) for p in parts]
    with GpuSph(int(off[-1]), G=1.0, theta=1.0e-4, leaf_size=8, multipole=1, max_neighbours=256, mac=mac, local_theta=0.0) as s:
        s.upload_batch(np.concatenate(parts), off, M.eos_table(), 0.1)
        for limit, flags in ((0, SORT_TIMEOUT), (DEFAULT_POLLS, SORT_TIMEOUT), (0, SORT_TIMEOUT)):
            _polls(s, limit)
            s.eval_forces()
            nb, g = s.neighbour_sets(), s.inspect("ACC_GRAV")[:, :3]
            d = s.diag(check=False)
            assert d["overflow_flags"] == flags and d["status"] == -4
            for k, n in enumerate(sizes):
                a = off[k]
                assert all(np.array_equal(nb[a + i], a + want[k][i]) for i in range(n))
                assert _rms(g[a:a + n], ref[k]) < 1e-5


def test_a_run_goes_on_through_a_sort_that_gave_up():
    n = 4000
    p = _cloud(n, 3)
    kw = dict(G=1.0, theta=1.0e-4, leaf_size=16, multipole=1, max_neighbours=256, local_theta=0.0)
    out = []
    for limit in (DEFAULT_POLLS, 0):
        with GpuSph(n, **kw) as s:
            s.upload(p, M.eos_table(), 0.1)
            s.set_dt(1e-3)
            s.encode_kdk(1)
            _polls(s, limit)
            s.encode_kdk(1)
            _polls(s, DEFAULT_POLLS)
            s.encode_kdk(2)
            out.append(s.readback())
    a, b = out
    for f in ("pos", "vel", "rho", "u"):  # the sums of some 10^2 neighbours in another order
        assert np.allclose(a[f], b[f], rtol=1e-4, atol=1e-4 * np.abs(a[f]).max()), f


def test_gravity_without_its_sort():
    n = 5000
    p = _cloud(n, 4)
    pos, mass = p["pos"].astype(np.float64), p["mass"].astype(np.float64)
    ref = oracle.gravity_direct64(pos, mass, 0.1, 1.0)
    with GpuSph(n, G=1.0, theta=1.0e-4, leaf_size=16, multipole=1) as s:
        for limit in (0, DEFAULT_POLLS):
            _polls(s, limit)
            assert _rms(s.gravity(pos, mass, 0.1, "tree"), ref) < 1e-5


def test_a_measurement_without_its_sort_fails_and_the_next_one_is_right():
    p = ds.scene(1)
    want = oracle.measure_disk(p, ds.G, variant=0)
    with GpuSph(len(p), G=ds.G, leaf_size=8) as s:
        s.upload(p, ds.eos(), 0.0)
        for _ in range(2):
            _polls(s, 0)
            with pytest.raises(SphError) as e:
                s.measure_disk(0)
            assert e.value.status == -4
            _polls(s, DEFAULT_POLLS)
            got = s.measure_disk(0)
            for k in ("clump_n", "n_clumps", "n_bound", "n_disk"):
                assert got[k] == want[k]
            assert got["disk_mass"] == pytest.approx(want["disk_mass"], rel=1e-9)
