"""The potential of the group walk at small softenings: a particle's own term, G m/ε, is no part of its potential and must
not pass through the running sum, where everything added after it would be rounded at its size. In both forms of the walk
(four warps to a group up to 32,768 particles, one above), with the accelerations and by itself.

Gravity with an opening angle near zero and no local expansion is the direct sum in f32. Tolerance: a sum of n positive terms good to
2^-24, rounded at random, is good to about 2^-25 sqrt(n) of itself: 1e-6 for 1,000, 6e-6 for 33,000 (RMS)."""
import numpy as np
import pytest

from botheadstudios_b200 import materials as M
from botheadstudios_b200.gpusph import GpuSph, particles_from_arrays

pytestmark = pytest.mark.gpu


def _phi64(pos, mass, eps, targets):
    out = np.empty(len(targets))
    for k, t in enumerate(targets):
        r = np.sqrt(((pos - pos[t]) ** 2).sum(1) + eps * eps)
        w = mass / r
        w[t] = 0.0
        out[k] = -w.sum()
    return out


@pytest.mark.parametrize("n,bound", [(1000, 1e-6), (33_000, 6e-6)])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("eps", [1e-1, 1e-4, 1e-5, 2e-6])
def test_potential_at_small_softenings(n, bound, precision, eps):
    rng = np.random.default_rng(n)
    pos = rng.normal(size=(n, 3))
    pos *= (rng.random(n) ** (1.0 / 3.0) / np.linalg.norm(pos, axis=1))[:, None]
    p = particles_from_arrays(pos, np.full(n, 1e-4), np.zeros((n, 3)), np.zeros(n), rng.uniform(0.5, 1.5, n),
                              np.zeros(n, np.uint32))
    x, m = p["pos"].astype(np.float64), p["mass"].astype(np.float64)
    tg = rng.choice(n, min(n, 500), replace=False)
    want = _phi64(x, m, np.float64(np.float32(eps)), tg)
    with GpuSph(n, G=1.0, theta=1e-4, leaf_size=16, multipole=1, max_neighbours=64, local_theta=0.0,
                precision=precision) as s:
        s.upload(p, M.eos_table(), eps)
        s.eval_forces()
        s.set_dt(1e-30)  # the particles stay
        for step in range(2):
            got = s.inspect("ACC_GRAV")[tg, 3].astype(np.float64)
            assert np.sqrt((((got - want) / want) ** 2).mean()) < bound, step
            s.encode_kdk(1)  # its walk leaves the potential out; the next look sums it alone
