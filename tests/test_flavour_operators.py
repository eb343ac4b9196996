"""The kkylin and rotate flavours are the same linear operators: the oracle's
restatements of both, applied to the same series for every translation a
tree produces (the M2L offsets, the M2M and L2L octants), agree to the
rounding of kkylin's recurrences (which divide by sin theta and multiply by
cot theta, at most 3.3 among the offsets, once per order m).  On the GPU both
flavours run the rotation kernels."""
import numpy as np
import pytest

# relative to the largest coefficient: 2.3e-16 times the recurrences' growth
TOL = {3: 1e-13, 8: 1e-12, 12: 1e-11, 16: 1e-10}


def multipole(oracle, c, p, rng):
    m = oracle.zeros_series(0, p)
    for _ in range(4):
        oracle.p2m(c + rng.uniform(-0.4, 0.4, 3), rng.uniform(-1, 1), c, p, out=m)
    return m


@pytest.mark.parametrize("p", sorted(TOL))
def test_m2l_offsets(oracle, p):
    rng = np.random.default_rng(p)
    codes = [(x, y, z) for x in range(-3, 4) for y in range(-3, 4) for z in range(-3, 4)
             if max(abs(x), abs(y), abs(z)) > 1]
    xs = np.array([0.3, -0.1, 0.2])
    m = multipole(oracle, xs, p, rng)
    for d in codes[:: 1 if p <= 8 else 5]:
        out = []
        for f in ("kkylin", "rotate"):
            lo = oracle.zeros_series(p, 0)
            oracle.to_local(f, (0, p), m, xs, (p, 0), lo, xs + np.array(d, float))
            out.append(np.array(lo))
        assert np.abs(out[0] - out[1]).max() <= TOL[p] * np.abs(out[1]).max(), d


@pytest.mark.parametrize("p", sorted(TOL))
def test_octants(oracle, p):
    rng = np.random.default_rng(100 + p)
    c = np.array([0.1, 0.2, -0.3])
    for o in range(8):
        t = np.array([0.5 if o & 1 else -0.5, 0.5 if o & 2 else -0.5, 0.5 if o & 4 else -0.5])
        m = multipole(oracle, c, p, rng)
        far = oracle.zeros_series(p, 0)
        oracle.p2l(c + np.array([3.0, -1.5, 2.0]), 1.0, c, p, out=far)
        for deg, src in (((0, p), m), ((p, 0), far)):
            out = []
            for f in ("kkylin", "rotate"):
                dst = oracle.zeros_series(*deg)
                oracle.translate(f, deg, src, c, deg, dst, c + t)
                out.append(np.array(dst))
            assert np.abs(out[0] - out[1]).max() <= TOL[p] * np.abs(out[1]).max(), (o, deg)
