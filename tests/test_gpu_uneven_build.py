"""Builds of unevenly spread points: nearly all of a segment falls into one bin of the
splitter's histogram, at one level or at many, so the median is selected from long
lists.  The tree is compared leaf by leaf with one built here by the split rule (cut at
rank n / 2 on the longest axis, ties in input order, leaves in order of x)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = {
    "uniform": lambda rng, n: rng.uniform(-50, 50, (n, 3)),
    "stray": lambda rng, n: np.r_[rng.uniform(1, 50, (n - 1, 3)), [[1e9, 2e9, 3e9]]],
    "strays": lambda rng, n: np.r_[rng.uniform(1, 50, (n - 40, 3)), rng.uniform(1e3, 1e9, (40, 3))],
    "towns": lambda rng, n: rng.uniform(1, 2, (n, 3)) + rng.integers(0, 4, (n, 1)) * 1e4,
    "tails": lambda rng, n: rng.standard_cauchy((n, 3)) * 5,
    "lattice": lambda rng, n: rng.integers(1, 13, (n, 3)),
    "equal": lambda rng, n: np.full((n, 3), 3.5),
    "heap": lambda rng, n: np.where(rng.random((n, 1)) < 0.6, 7.0, rng.uniform(1, 50, (n, 3))),
    "two": lambda rng, n: np.c_[rng.integers(1, 3, (n, 2)), np.ones(n)],
}


def leaves(pts, fill):
    """Point numbers in the order of the tree's leaves."""
    out, todo = [], [np.arange(len(pts))]
    while todo:
        i = todo.pop()
        if len(i) <= fill:
            out.append(i[np.argsort(pts[i, 0], kind="stable")])
            continue
        p = pts[i]
        ext = p.max(0) - p.min(0)
        axis = int(np.argmax(ext))
        left = np.zeros(len(i), bool)
        left[np.argsort(p[:, axis], kind="stable")[:len(i) // 2]] = True
        todo += [i[~left], i[left]]
    return np.concatenate(out)


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("n", [4097, 9001, 140001, 700001])
def test_leaves_follow_the_split_rule(ikdg_mod, n, kind):
    pts = KINDS[kind](np.random.default_rng(n), n).astype(np.float32)
    tree = ikdg_mod.KDTree()
    tree.set_leaf_fill(32)
    tree.Build(pts)
    assert tree.validate() == 0
    big = np.float32(3e38)
    ids = tree.box_search(np.array([[-big, -big, -big, big, big, big]]))[1]
    assert np.array_equal(ids, leaves(pts, 32))
    tree.close()
