"""The point-set walk (sph_gravity, sph_gravity_tree_noalloc) at the edges of its tiles: blocks of 32 points, rounds of
128 nodes, leaves with and without halves, partial last leaves and coincident points.

The reference is the walk's definition restated in f64 on the tree that the context reports: every point opens nodes
for itself, leaves of 16 and more are accepted or summed by halves. Tolerance: the device adds at most 4,097 terms of
f32 arithmetic, each good to a few 2^-24, so 1e-5 RMS (an opening decision within f32 rounding of its limit may go
the other way; a few such nodes among two million change the RMS by less)."""
import math

import numpy as np
import pytest

from botheadstudios_b200 import materials as M
from botheadstudios_b200.gpusph import GpuSph, particles_from_arrays
from refcases import cloud

pytestmark = pytest.mark.gpu
G = 6.674e-11
SOFT = 5.0e3


def _moments(x, m, quad):
    """Mass, centre of mass and traceless quadrupole of a run of points."""
    M0 = m.sum()
    com = (m[:, None] * x).sum(0) / M0
    d = x - com
    Q = (m[:, None, None] * (3.0 * d[:, :, None] * d[:, None, :] - (d * d).sum(1)[:, None, None] * np.eye(3))).sum(0)
    return M0, com, Q if quad else np.zeros((3, 3))


def _multipole(d, M0, Q):
    r2 = (d * d).sum(1) + SOFT**2
    r = np.sqrt(r2)
    e = d / r[:, None]
    Qe = e @ Q
    eQe = (e * Qe).sum(1)
    return G * (M0 / r2[:, None] * e + (2.5 * eQe[:, None] * e - Qe) / (r2 * r2)[:, None])


def _pairs(x, src, ms, self_at):
    d = src[None] - x[:, None]
    r2 = (d * d).sum(2) + SOFT**2
    w = G * ms[None] / (r2 * np.sqrt(r2))
    w[self_at >= 0, self_at[self_at >= 0]] = 0.0
    return (w[:, :, None] * d).sum(1)


def _walk(t, x, m, leaf, quad, theta):
    """Accelerations of the sorted points x by their own walks over the tree t."""
    n, L = len(x), t["L"]
    half = leaf // 2 if leaf >= 16 else 0
    acc = np.zeros((n, 3))

    def span(node):  # the sorted points under a node
        a = b = node
        while a < L - 1:
            a = t["LEFT"][a]
        while b < L - 1:
            b = t["RIGHT"][b]
        return (a - (L - 1)) * leaf, min((b - (L - 1) + 1) * leaf, n)

    stack = [(0, np.arange(n))]
    while stack:
        node, who = stack.pop()
        p = x[who]
        com, lo, hi = t["COM"][node, :3], t["LO"][node, :3], t["HI"][node]
        d = com - p
        inside = ((lo <= p) & (p <= hi[:3])).all(1)
        take = ~inside & ((d * d).sum(1) + SOFT**2 >= (hi[3] * 1.00001) ** 2)
        s0, s1 = span(node)
        if take.any():
            M0, c, Q = _moments(x[s0:s1], m[s0:s1], quad)
            acc[who[take]] += _multipole(c - p[take], M0, Q)
        rest, rp, rin = who[~take], p[~take], inside[~take]
        if not len(rest):
            continue
        if node < L - 1:
            stack += [(t["LEFT"][node], rest), (t["RIGHT"][node], rest)]
            continue
        for a in range(s0, s1, half or leaf):
            b = min(a + (half or leaf), s1)
            far = np.zeros(len(rest), bool)
            if half:
                M0, c, Q = _moments(x[a:b], m[a:b], quad)
                mid, size = 0.5 * (x[a:b].min(0) + x[a:b].max(0)), (x[a:b].max(0) - x[a:b].min(0)).max()
                ro = (size / theta + np.linalg.norm(mid - c)) * 1.00001
                d = c - rp
                far = ~rin & ((d * d).sum(1) + SOFT**2 >= ro * ro)
                acc[rest[far]] += _multipole(d[far], M0, Q)
            near = rest[~far]
            self_at = np.where((near >= a) & (near < b), near - a, -1)
            acc[near] += _pairs(x[near], x[a:b], m[a:b], self_at)
    return acc


@pytest.mark.parametrize("n", [1, 2, 31, 33, 64, 1000, 4097])
@pytest.mark.parametrize("leaf,quad", [(1, 0), (8, 1), (16, 0), (16, 1), (32, 1)])
def test_point_walk_matches_its_definition(n, leaf, quad):
    _, pos, mass = cloud(n, 31 + n)
    if n > 64:
        pos[n // 2:n // 2 + 40] = pos[n // 2]  # coincident points: no force between them, one Morton code
    pos, mass = pos.astype(np.float32).astype(np.float64), mass.astype(np.float32).astype(np.float64)
    parts = particles_from_arrays(pos, np.ones(n), np.zeros((n, 3)), np.zeros(n), mass, np.zeros(n, np.uint32))
    for theta in (1.0e-4, 0.5):
        with GpuSph(n, G=G, theta=theta, leaf_size=leaf, multipole=quad, max_neighbours=64) as s:
            got = s.gravity(pos, mass, SOFT, "tree")
            s.upload(parts, M.eos_table(), SOFT)
            s.eval_forces()  # the context's own tree over the same points: what the reference walks
            t = dict(L=s.n_leaves(), LEFT=s.inspect("LEFT"), RIGHT=s.inspect("RIGHT"),
                     COM=s.inspect("NODE_COM").astype(np.float64), LO=s.inspect("NODE_BMIN").astype(np.float64),
                     HI=s.inspect("NODE_BMAX").astype(np.float64))
            order = s.inspect("ORDER")
        want = np.empty_like(got)
        want[order] = _walk(t, pos[order], mass[order], leaf, quad, np.float64(np.float32(theta)))
        assert np.isfinite(got).all()
        err = math.sqrt(((got - want) ** 2).sum() / max((want**2).sum(), 1e-300))
        assert err < 1e-5, (theta, err)


def test_allocation_free_calls_in_a_row_leave_the_scratch_as_they_found_it():
    """Every call resets what the sort and the tree keep between calls, so any sequence of sizes repeats its results."""
    import ctypes as C

    import torch

    from botheadstudios_b200 import _lib

    L = _lib.load()
    first = {}
    for n in (65_536, 33, 20_000, 65_536, 1, 33, 1_025, 20_000, 1_025, 1, 65_536):
        _, pos, mass = cloud(n, 77)
        body = torch.tensor(np.concatenate([pos, mass[:, None]], 1).astype(np.float32), device="cuda:0")
        out = torch.full((n, 4), float("nan"), dtype=torch.float32, device="cuda:0")
        s = torch.cuda.current_stream(0)
        assert L.sph_gravity_tree_noalloc(C.c_void_p(body.data_ptr()), n, G, SOFT, 0.5, 8, 1, C.c_void_p(out.data_ptr()),
                                          C.c_void_p(s.cuda_stream)) == _lib.SPH_OK
        s.synchronize()
        a = out.cpu().numpy()
        assert np.isfinite(a).all()
        assert np.array_equal(a, first.setdefault(n, a))
