"""The Morton sort at the edges of its tiles and of its two forms (one launch with tiles of 1,024 and 2,048 keys, the
chain of launches above 303,104): codes as the reference quantises them, order by (impact, code, original index),
exactly, also on the next sort out of the same workspace and for a batch."""
import numpy as np
import pytest

from botheadstudios_b200 import materials as M
from botheadstudios_b200.gpusph import GpuSph, particles_from_arrays

pytestmark = pytest.mark.gpu


def _codes(pos):
    """Morton codes in f32 (bh_gravity.wgsl:91-108)."""
    lo = pos.min(0)
    ext = np.maximum(pos.max(0) - lo, np.float32(1e-30))
    q = np.clip(np.floor(np.clip((pos - lo) / ext, 0, 1).astype(np.float32) * np.float32(1024)), 0, 1023).astype(np.uint64)
    code = np.zeros(len(pos), np.uint64)
    for b in range(10):
        for a in range(3):
            code |= ((q[:, a] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + 2 - a)
    return code


def _parts(n, seed):
    rng = np.random.default_rng(seed)
    pos = rng.normal(size=(n, 3)).astype(np.float32)
    pos[rng.random(n) < 0.3] *= np.float32(1e-3)  # a dense core: runs of equal codes longer than a tile
    return particles_from_arrays(pos, np.full(n, 1e-6), np.zeros((n, 3)), np.zeros(n), np.ones(n), np.zeros(n, np.uint32))


def _check(s, parts, offsets):
    s.eval_forces()
    codes, order = s.inspect("CODES"), s.inspect("ORDER")
    assert s.diag()["overflow_flags"] == 0
    for a, b in zip(offsets[:-1], offsets[1:]):
        want = _codes(parts["pos"][a:b])
        o = np.argsort(want, kind="stable")
        assert np.array_equal(order[a:b], a + o)
        assert np.array_equal(codes[a:b], want[o])


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 2049, 65_536, 65_537, 303_104, 303_105])
def test_sort_is_exact_at_the_edges_of_its_tiles(n):
    with GpuSph(n, gravity="none", leaf_size=16, max_neighbours=4) as s:
        for seed in (n, n + 1):
            p = _parts(n, seed)
            s.upload(p, M.eos_table(), 0.0)
            _check(s, p, [0, n])


@pytest.mark.parametrize("sizes", [[1, 1500, 33, 1024], [200_000, 7, 103_200]])
def test_sort_of_a_batch_keeps_the_impacts_apart(sizes):
    offsets = np.concatenate([[0], np.cumsum(sizes)])
    p = _parts(int(offsets[-1]), 5)
    with GpuSph(len(p), gravity="none", leaf_size=16, max_neighbours=4) as s:
        s.upload_batch(p, offsets, M.eos_table(), 0.0)
        _check(s, p, offsets)


@pytest.mark.parametrize("n", [5_000, 100_000])
def test_sorts_in_a_row_stay_exact(n):
    """Many blocks leave the ticket loop at different times, many times."""
    p = _parts(n, 9)
    with GpuSph(n, gravity="none", leaf_size=16, max_neighbours=4) as s:
        s.upload(p, M.eos_table(), 0.0)
        for _ in range(60):
            _check(s, p, [0, n])


def test_one_workspace_sorts_by_both_forms_in_turn():
    """A context is refilled with fewer particles: the chain's counts must not pass for the one launch's tile words."""
    with GpuSph(400_000, gravity="none", leaf_size=16, max_neighbours=4) as s:
        for n in (400_000, 50_000, 200_000, 400_000, 300_000, 60_000, 304_000, 1_500, 303_104):
            p = _parts(n, n + 3)
            s.upload(p, M.eos_table(), 0.0)
            _check(s, p, [0, n])
