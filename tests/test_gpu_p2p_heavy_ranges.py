"""The mixed near field where the first 32 near ranges of a leaf are all heavy
(left to the chunked pass) and more follow: an empty batch of ranges, then one
that is not, against the FP64 direct sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MAXBOX = 4096
HEAVY, LIGHT = 2100, 100     # points of a cell: above and below kBigRange


def cells():
    """Points per cell (edge 1/4, or 1/8 for the eight children of cell (1, 1,
    1)): the 8 children, 24 heavy neighbours, then the two light neighbours that
    come last in node order, and cells that keep the octants divided."""
    out = [((2 + i, 2 + j, 2 + k), 0.125, HEAVY) for k in (0, 1) for j in (0, 1) for i in (0, 1)]
    for k in range(3):
        for j in range(3):
            for i in range(3):
                if (i, j, k) != (1, 1, 1):
                    light = (i, j, k) in ((1, 2, 2), (2, 2, 2))
                    out.append(((i, j, k), 0.25, LIGHT if light else HEAVY))
    return out + [((0, 3, 3), 0.25, HEAVY), ((3, 3, 3), 0.25, MAXBOX)]


@pytest.mark.parametrize("field", [False, True])
def test_first_ranges_all_heavy(aran, oracle, field):
    rng = np.random.default_rng(11)
    x = np.concatenate([(np.array(c) + rng.uniform(0.0, 1.0, (n, 3))) * h for c, h, n in cells()])
    q = rng.uniform(0.0, 1.0, len(x))
    targets = rng.choice(8 * HEAVY, 400, replace=False)       # in the eight children
    with aran.Solver3d(maxbox=MAXBOX, order=12, field=field, precision="mixed") as s:
        pot, fld = s.solve(x, q)
        info, lists = s.tree_info(), s.tree_lists()
    # each of the eight children: 32 heavy ranges, then the light ones
    size = dict(zip(lists["ids"].tolist(), (lists["end"] - lists["begin"]).tolist()))
    leaf, count = np.unique(lists["near"][:, 0], return_counts=True)
    assert info["depth"] == 3 and (count == 34).sum() == 8
    for row in leaf[count == 34]:
        got = [size[int(b)] for a, b in lists["near"] if a == row]
        assert min(got[:32]) == HEAVY and got[32:] == [LIGHT, LIGHT]
    rp, rf = oracle.direct(x, q, targets=targets)
    # one sign: the potential is good to the truncation of order 12, 3e-7, times a margin
    assert np.linalg.norm(pot[targets] - rp) < 2e-6 * np.linalg.norm(rp)
    if field:
        assert np.linalg.norm(fld[targets] - rf) < 2e-5 * np.linalg.norm(rf)
