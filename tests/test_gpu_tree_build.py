"""The group walk's tree at the edges of the builder's runs of leaves (128 with up to 32 to either side): links in Karras
numbering over the index-extended codes, exactly; boxes exactly; masses to f32 rounding (at most 2,000 terms: 1e-5).
Clouds with a dense core give runs of equal codes longer than a run of leaves; a batch gives several subtrees."""
import numpy as np
import pytest

from botheadstudios_b200 import materials as M
from botheadstudios_b200.gpusph import GpuSph, particles_from_arrays

pytestmark = pytest.mark.gpu


def _links(keys):
    """(left, right, parent) of the radix tree over distinct sorted keys (Python ints), root 0, a left child numbered by
    its last leaf and a right child by its first."""
    L = len(keys)
    left, right, parent = [0] * max(L - 1, 0), [0] * max(L - 1, 0), [0xFFFFFFFF] * (2 * L - 1)
    todo = [(0, L - 1, 0)]
    while todo:
        a, b, node = todo.pop()
        if a == b:
            continue
        top = (keys[a] ^ keys[b]).bit_length() - 1
        lo, hi = a, b  # the first leaf with that bit set
        while hi - lo > 1:
            mid = (lo + hi) // 2
            if (keys[mid] >> top) & 1:
                hi = mid
            else:
                lo = mid
        for x, y, own, out in ((a, lo, lo, left), (hi, b, hi, right)):
            child = L - 1 + x if x == y else own
            out[node] = child
            parent[child] = node
            todo.append((x, y, child))
    return left, right, parent


def _check(sizes, K, dense, seed):
    rng = np.random.default_rng(seed)
    n = sum(sizes)
    pos = rng.normal(size=(n, 3)).astype(np.float32)
    pos[rng.random(n) < dense] *= np.float32(1e-4)
    mass = rng.uniform(0.5, 1.5, n).astype(np.float32)
    h = rng.uniform(1e-6, 2e-6, n).astype(np.float32)
    p = particles_from_arrays(pos, h, np.zeros((n, 3)), np.zeros(n), mass, np.zeros(n, np.uint32))
    off = np.concatenate([[0], np.cumsum(sizes)])
    with GpuSph(n, gravity="none", leaf_size=K, max_neighbours=4) as s:
        for _ in range(2):  # the second build finds the workspace as the first one left it
            s.upload_batch(p, off, M.eos_table(), 0.0)
            s.eval_forces()
        left, right, parent = s.inspect("LEFT"), s.inspect("RIGHT"), s.inspect("PARENT")
        com, lo, hi = s.inspect("NODE_COM"), s.inspect("NODE_BMIN"), s.inspect("NODE_BMAX")
        codes, order = s.inspect("CODES"), s.inspect("ORDER")
    starts, keys = [], []
    for k in range(len(sizes)):
        for j, a in enumerate(range(off[k], off[k + 1], K)):
            starts.append(a)
            keys.append((k << 62) | (int(codes[a]) << 32) | j)
    L = len(starts)
    want = _links(keys)
    assert np.array_equal(left, want[0]) and np.array_equal(right, want[1]) and np.array_equal(parent, want[2])
    bmin, bmax = np.empty((2 * L - 1, 4), np.float32), np.empty((2 * L - 1, 3), np.float32)
    m = np.empty(2 * L - 1)
    ends = starts[1:] + [n]
    for c in range(L):
        who = order[starts[c]:min(ends[c], starts[c] + K)]
        bmin[L - 1 + c] = (*pos[who].min(0), h[who].max())
        bmax[L - 1 + c] = pos[who].max(0)
        m[L - 1 + c] = mass[who].astype(np.float64).sum()
    done = []
    todo = [0] if L > 1 else []
    while todo:
        i = todo.pop()
        done.append(i)
        todo += [x for x in (left[i], right[i]) if x < L - 1]
    for i in reversed(done):
        a, b = left[i], right[i]
        bmin[i] = (*np.minimum(bmin[a, :3], bmin[b, :3]), max(bmin[a, 3], bmin[b, 3]))
        bmax[i], m[i] = np.maximum(bmax[a], bmax[b]), m[a] + m[b]
    assert np.array_equal(lo, bmin) and np.array_equal(hi[:, :3], bmax)
    assert np.allclose(com[:, 3], m, rtol=1e-5)


@pytest.mark.parametrize("L", [1, 2, 95, 96, 97, 128, 129, 160, 161, 192, 257, 1000])
@pytest.mark.parametrize("K,dense", [(1, 0.0), (1, 0.9), (32, 0.3)])
def test_tree_at_the_edges_of_the_runs(L, K, dense):
    _check([L * K - (K // 2 if L > 1 else 0)], K, dense, L + K)


def test_tree_of_a_batch():
    _check([40, 1, 300, 129, 7, 513], 2, 0.5, 3)
