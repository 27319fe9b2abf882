"""The hi/lo mode's compensated sums where four warps share a group (up to 32,768 particles): the warps' sums are added with
their compensations, so that a component is rounded once, at its end.

A particle at the origin between the corners (±1, ±1, ±1), softening 1: R² = 4 for every other particle, so a term is a mass
over eight, an exact number, and the sum is a whole number of eighths. Smoothing lengths that reach everything keep all
leaves on the pairwise list. Equal masses at opposite corners cancel; a few odd ones remain, so the warps' shares (some
2^29 each) are larger than the sum (2^25). Tolerance: a compensated sum of n terms is off by n 2^-48 Σ|term| = 0.1 at most
(Higham, Accuracy and Stability of Numerical Algorithms, §4.3) before its last rounding, 2 here; 4 leaves room for both.
Rounded shares would be off by some 2^5."""
import numpy as np
import pytest

from botheadstudios_b200 import materials as M
from botheadstudios_b200.gpusph import GpuSph, particles_from_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf", [1, 8])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_compensated_sums_are_rounded_once(leaf, seed):
    rng = np.random.default_rng(seed)
    pairs = 2000
    corner = rng.choice([-1.0, 1.0], (pairs, 3))
    mass = rng.integers(1 << 22, 1 << 24, pairs).astype(np.float64)
    odd = np.array([[1, 1, 1], [1, -1, 1], [-1, 1, 1]], np.float64)
    pos = np.concatenate([np.zeros((1, 3)), corner, -corner, odd])
    m = np.concatenate([[1.0], mass, mass, np.array([37.0 * 2**23, 11.0 * 2**22, 5.0 * 2**22 + 4.0])])
    n = len(m)
    p = particles_from_arrays(pos, np.full(n, 4.0), np.zeros((n, 3)), np.zeros(n), m, np.zeros(n, np.uint32))
    with GpuSph(n, G=1.0, theta=0.5, leaf_size=leaf, multipole=0, max_neighbours=4096, local_theta=0.0, precision=1) as s:
        s.upload(p, M.eos_table(), 1.0)
        s.eval_forces()
        got = s.inspect("ACC_GRAV")[0, :3].astype(np.float64)
    want = (m[:, None] * pos / 8.0).sum(0)
    assert np.abs(got - want).max() <= 4.0, (got, want)
