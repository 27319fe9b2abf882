"""The point-set walk (sph_gravity, sph_gravity_tree_noalloc) at the edges of its tiles: blocks of 32 points, rounds of
128 nodes, leaves with and without halves, partial last leaves and coincident points, against the FP64 direct sum.

Tolerances: with θ → 0 every pair is summed in f32, whose terms are good to a few 2^-24 and whose sums run over at
most 4,097 of them, so 1e-5 RMS; at θ = 0.5 the tree's truncation decides, 1e-2 as for the context's other point-set
checks."""
import math

import numpy as np
import pytest

import oracle
from botheadstudios_b200.gpusph import GpuSph
from refcases import cloud

pytestmark = pytest.mark.gpu
G = 6.674e-11
SOFT = 5.0e3


def _rms(a, ref):
    return math.sqrt(((a - ref) ** 2).sum() / max((ref ** 2).sum(), 1e-300))


@pytest.mark.parametrize("n", [1, 2, 31, 33, 64, 1000, 4097])
@pytest.mark.parametrize("leaf,quad", [(1, 0), (8, 1), (16, 0), (16, 1), (32, 1)])
def test_point_walk_against_direct_sum(n, leaf, quad):
    _, pos, mass = cloud(n, 31 + n)
    if n > 64:
        pos[n // 2:n // 2 + 40] = pos[n // 2]  # coincident points: no force between them, one Morton code
    ref = oracle.gravity_direct64(pos, mass, SOFT, G)
    for theta, bound in ((1.0e-4, 1e-5), (0.5, 1e-2)):
        with GpuSph(n, G=G, theta=theta, leaf_size=leaf, multipole=quad) as s:
            a = s.gravity(pos, mass, SOFT, "tree")
        assert np.isfinite(a).all()
        assert _rms(a, ref) < bound, (theta, _rms(a, ref))
