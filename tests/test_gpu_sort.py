"""The key sort under the octree at the sizes where its form changes (ranks by
comparison, radix tiles of 1,024, 2,048 and 4,096 keys, partial tiles and
groups), through the tree it numbers: node ranges against a numpy sort of the
same keys, and run-to-run identical nodes."""
import numpy as np
import pytest

from conftest import E

pytestmark = pytest.mark.gpu


def _expected_ranges(x, y, z, cap):
    """(begin, end) of every node of the reference's octree, any order."""
    p = [x, y, z]
    lo, hi = [a.min() for a in p], [a.max() for a in p]
    h = 0.5 * max(b - a for a, b in zip(lo, hi)) * (1.0 + 1e-9)
    c = [np.full(len(x), 0.5 * (a + b)) for a, b in zip(lo, hi)]
    key = np.zeros(len(x), np.uint64)
    for _ in range(21):
        bits = [a >= b for a, b in zip(p, c)]
        key = (key << np.uint64(3)) | sum(b.astype(np.uint64) << np.uint64(d) for d, b in enumerate(bits))
        h *= 0.5
        c = [a + np.where(b, h, -h) for a, b in zip(c, bits)]
    key.sort()
    ranges, parents = [(0, len(x))], [(0, len(x))]
    for d in range(1, 22):
        pre = key >> np.uint64(3 * (21 - d))
        level = []
        for b, e in parents:
            if e - b <= cap:
                continue
            cut = np.concatenate([[b], b + 1 + np.nonzero(pre[b + 1:e] != pre[b:e - 1])[0], [e]])
            level += list(zip(cut[:-1].tolist(), cut[1:].tolist()))
        ranges += level
        parents = level
    return sorted(ranges)


@pytest.mark.parametrize("n", [1, 255, 257, 1024, 1025, 16384, 16385, 17408, 150000, 150001, 600000, 600001])
def test_tree_ranges(sim, n):
    rng = np.random.default_rng(n)
    x, y, z = rng.normal(0.0, [[1e-4], [1e-4], [3e-4]], (3, n))
    if n > 100:  # equal keys: duplicates keep their input order
        x[: n // 50], y[: n // 50], z[: n // 50] = x[-(n // 50):], y[-(n // 50):], z[-(n // 50):]
    cap = 8 if n < 50000 else 64
    f, g = sim.bh_tree(x, y, z, np.full(n, E), leaf_capacity=cap)
    assert sorted(zip(g[:, 8].tolist(), g[:, 9].tolist())) == _expected_ranges(x, y, z, cap)
    f2, g2 = sim.bh_tree(x, y, z, np.full(n, E), leaf_capacity=cap)
    assert np.array_equal(f, f2) and np.array_equal(g, g2)
