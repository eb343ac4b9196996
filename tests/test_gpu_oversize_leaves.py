"""Leaves above the capacity (the depth limit keeps them): the near field takes them
by several blocks, against the direct sum; its time does not hang on the capacity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def one_octant(n, seed):
    """n points in the first octant of the box and one far from it."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.0, 0.4, (n + 1, 3))
    x[n] = 0.9
    return x, rng.uniform(-1.0, 1.0, n + 1)


SIZES = [17, 64, 65, 128, 129, 700, 2049, 4200]


@pytest.mark.parametrize("n", SIZES)
def test_mixed_against_the_direct_sum(aran, n):
    x, q = one_octant(n, n)
    d = x[:, None] - x[None]
    r = np.sqrt((d ** 2).sum(-1))
    np.fill_diagonal(r, np.inf)
    w = q / r
    tol = 2e-6                 # a pair: offset, reciprocal square root
    for field in (False, True):
        with aran.Solver3d(maxbox=16, order=4, field=field, precision="mixed", max_depth=1) as s:
            pot, fld = s.solve(x, q)
        assert np.all(np.abs(pot - w.sum(1)) <= tol * np.abs(w).sum(1))
        if field:
            g = -((w / r ** 2)[:, :, None] * d).sum(1)
            assert np.all(np.abs(fld - g) <= 3 * tol * np.abs(w / r).sum(1)[:, None])


@pytest.mark.parametrize("n", SIZES)
def test_fp64_against_the_oracle(aran, oracle, n):
    x, q = one_octant(n, n)
    with aran.Solver3d(maxbox=16, order=4, precision="fp64", max_depth=1) as s:
        pot, fld = s.solve(x, q)
    rp, rf = oracle.direct(x, q)
    assert np.linalg.norm(pot - rp) < 1e-12 * np.linalg.norm(rp)   # as the other FP64 tests
    assert np.linalg.norm(fld - rf) < 1e-12 * np.linalg.norm(rf)


def test_time_at_small_capacities(aran):
    """A leaf of 6,000 points costs the same at capacities 16 and 64, whose kernels
    have blocks of 64 and 128 threads (half as much again is allowed)."""
    x, q = one_octant(6000, 1)
    ms = {}
    for maxbox in (16, 64):
        with aran.Solver3d(maxbox=maxbox, order=4, precision="mixed", max_depth=1) as s:
            t = []
            for _ in range(4):
                s.solve(x, q)
                t.append(s.timings()["p2p"])
        ms[maxbox] = min(t)
    assert ms[16] < 1.5 * ms[64], ms


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [9, 32, 33, 128, 129, 700, 4200])
def test_2d_against_the_direct_sum(aran, oracle, n, precision):
    rng = np.random.default_rng(n)
    x = rng.uniform(-0.9, -0.1, (n + 1, 2))
    x[n] = 0.8
    q = rng.uniform(-1.0, 1.0, n + 1)
    z = x[:, 0] + 1j * x[:, 1]
    d = z[:, None] - z[None]
    np.fill_diagonal(d, np.inf)
    with aran.Solver2d(maxbox=8, order=8, precision=precision, max_depth=1) as s:
        a = s.solve(x, q)
    if precision == "mixed":   # a pair: offset and reciprocal, as in 3D
        assert np.all(np.abs(a - (q / d).sum(1)) <= 2e-6 * np.abs(q / d).sum(1))
    else:
        ref = oracle.direct2d(x, q)
        assert np.linalg.norm(a - ref) < 1e-12 * np.linalg.norm(ref)


def test_2d_time_at_small_capacities(aran):
    x = np.random.default_rng(2).uniform(-0.9, -0.1, (6000, 2))
    q = np.ones(len(x))
    ms = {}
    for maxbox in (8, 200):
        with aran.Solver2d(maxbox=maxbox, order=8, precision="mixed", max_depth=1) as s:
            t = []
            for _ in range(4):
                s.solve(x, q)
                t.append(s.timings()["p2p"])
        ms[maxbox] = min(t)
    assert ms[8] < 1.5 * ms[200], ms
