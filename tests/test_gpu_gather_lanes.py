"""The density sums with two and with four lanes to a particle (the choice goes by the size of the whole batch, with a
line at 20,000 particles) give the same bits: an impact alone and beside others that take the batch across the line. Lists of no entry, of fewer than a chunk and of several chunks; the solve's odd and even passes."""
import numpy as np
import pytest

from botheadstudios_b200 import materials as M
from botheadstudios_b200.gpusph import GpuSph, particles_from_arrays

pytestmark = pytest.mark.gpu


def _cloud(n, seed, h=1.7):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0.0, n ** (1.0 / 3.0), (n, 3)).astype(np.float32)
    vel = rng.normal(0.0, 0.05, (n, 3))
    return particles_from_arrays(pos, np.full(n, h) * rng.uniform(0.5, 1.2, n), vel, np.full(n, 1e3),
                                 rng.uniform(0.5, 1.5, n), np.zeros(n, np.uint32))


def _run(parts, **kw):
    off = np.concatenate([[0], np.cumsum([len(p) for p in parts])])
    with GpuSph(int(off[-1]), G=1.0, theta=0.6, leaf_size=16, multipole=1, max_neighbours=256, **kw) as s:
        s.upload_batch(np.concatenate(parts), off, M.eos_table(), 0.1)
        s.set_dt(1e-4)
        s.encode_kdk(2)
        assert s.diag()["overflow_flags"] == 0
        return s.readback()


@pytest.mark.parametrize("kw", [dict(h_mode=0), dict(h_mode=0, kernel="wendland"), dict(h_mode=1, h_iters=1),
                                dict(h_mode=1, h_iters=2, kernel="wendland"), dict(h_mode=1, h_iters=3),
                                dict(h_mode=2, h_iters=2, kernel="wendland"), dict(h_mode=0, block_threads=96)],
                         ids=lambda k: "-".join(str(v) for v in k.values()))
def test_any_number_of_lanes_gives_the_same_bits(kw):
    if kw["h_mode"]:
        kw = dict(kw, h_neighbours=32.0)
    parts = [_cloud(n, n) for n in (1, 3, 33, 4099, 19_990)]
    alone = np.concatenate([_run([p], **kw) for p in parts])  # four lanes each
    for filler in (10_000, 180_000):                          # then two
        got = _run(parts + [_cloud(filler, 5)], **kw)[: len(alone)]
        for f in got.dtype.names:
            assert np.array_equal(got[f], alone[f]), (filler, f)
