"""Box deletions whose boxes differ much in size: a large box among many passes most of
its subtrees on to a second launch, and with many large ones the list of those is full.
Counts, the points that are left and the structure are those of the boxes applied to
all points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(3000, 40), (3000, 2500), (200000, 40), (200000, 300), (200000, 2500), (1000003, 300)])
@pytest.mark.parametrize("kind", ["one_large", "all_large", "everything", "nested", "none"])
def test_large_boxes_among_many(ikdg_mod, n, m, kind):
    rng = np.random.default_rng(n + m)
    pts = rng.uniform(-20, 20, (n, 3)).astype(np.float32)
    tree = ikdg_mod.KDTree(0.999, 0.999, 0.5)
    tree.Build(pts)
    c = rng.uniform(-20, 19, (m, 3))
    s = rng.uniform(0.05, 0.6, (m, 3))
    b = np.concatenate([c, c + s], 1)
    if kind == "one_large":
        b[m // 2] = [-20, -20, -3, 20, 7, 20]
    elif kind == "all_large":
        b = np.concatenate([rng.uniform(-20, -5, (m, 3)), rng.uniform(5, 20, (m, 3))], 1)
    elif kind == "everything":
        b[::m // 3] = [-21, -21, -21, 21, 21, 21]
    elif kind == "nested":
        h = np.linspace(0.1, 18, m)[:, None]
        b = np.concatenate([np.repeat(-h, 3, 1), np.repeat(h, 3, 1)], 1)
    else:
        b += 100
    b = b.astype(np.float32)
    gone = np.zeros(n, bool)
    by_x = np.argsort(pts[:, 0])
    xs = pts[by_x, 0]
    for x in b:
        i = by_x[np.searchsorted(xs, x[0]):np.searchsorted(xs, x[3])]
        i = i[~gone[i]]
        p = pts[i]
        gone[i[((p >= x[:3]) & (p < x[3:])).all(1)]] = True
    assert tree.Delete_Point_Boxes(b) == gone.sum()
    assert tree.validate() == 0 and tree.validnum() == n - gone.sum()
    assert np.array_equal(np.sort(tree.flatten(with_ids=True)[1]), np.flatnonzero(~gone))
    assert tree.Delete_Point_Boxes(b) == 0
    tree.close()
