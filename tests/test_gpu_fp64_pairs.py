"""The FP64 kernels' pair terms where they can go wrong: tile remainders in
every lane shape, tied nearest neighbours, and squared distances outside the
normal range (coincident particles, separations whose square is subnormal or
overflows), against the FP64 oracle.

Tolerance: each side's sum of n terms is within (n + 40) u sum|term| of the
exact one (u = 2^-53; 40 covers a term's own roundings), so the two differ
by at most twice that.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_cid = [7100]


def engine(npipes=4096):
    from starlab_b200 import G6Engine
    _cid[0] += 1
    return G6Engine(cluster_id=_cid[0], precision="fp64", npipes=npipes)


def cluster(n, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(0.1, 1.0, n) / n, rng.normal(size=(n, 3)), rng.normal(size=(n, 3))


def run(m, x, v, members, eps2, index=None, h2=None):
    n = len(m)
    eng = engine()
    z = np.zeros((n, 3))
    eng.set_j_particles(0.0, m, z, z, v, x, index=index)
    eng.set_ti(0.0)
    idx = (np.arange(n) if index is None else index)[members].astype(np.int32)
    eng.calc_firsthalf(n, idx, x[members], v[members], eps2, h2)
    out = eng.calc_lasthalf2()
    eng.close()
    return out


def bounds(m, x, v, members, eps2):
    """2 (n + 40) u sum|term| for acc, jerk (per component: the vector's) and pot."""
    n = len(m)
    d, dv = x[None] - x[members, None], v[None] - v[members, None]
    r2 = (d * d).sum(2) + eps2
    r2[np.arange(len(members)), members] = np.inf
    r2 = np.where(r2 == 0, np.inf, r2)
    w = m / r2 ** 1.5
    top = np.maximum(np.abs(d).max(2), 1e-300)  # |d| without overflow
    dl, vl = top * np.sqrt(((d / top[..., None]) ** 2).sum(2)), np.sqrt((dv * dv).sum(2))
    f = 2 * (n + 40) * 2.0 ** -53
    return f * (w * dl).sum(1), f * (w * vl * 4.0).sum(1), f * (m / np.sqrt(r2)).sum(1)


def check(got, ref, tol, rows=None):
    rows = slice(None) if rows is None else rows
    for k, q in enumerate(("acc", "jerk", "pot")):
        d = np.abs(got[k][rows] - ref[k][rows])
        t = tol[k][rows]
        assert np.all(d <= (t[:, None] if d.ndim == 2 else t)), (q, float((d.max(-1) / t).max()))


# n around the 128-j tile and the runs of 8 and 16 records; ni in the shapes
# of one, eight and thirty-two i per warp, and two i per thread (8192 up)
@pytest.mark.parametrize("n,ni", [(2, 1), (3, 2), (9, 8), (127, 9), (128, 31), (129, 33), (257, 2), (1000, 17),
                                  (1025, 300), (2049, 700), (8200, 8193)])
@pytest.mark.parametrize("eps2", [0.0, 1e-4])
def test_sizes(oracle, n, ni, eps2):
    m, x, v = cluster(n, 31 * n + ni)
    members = np.sort(np.random.default_rng(n).choice(n, ni, replace=False))
    if ni > 1000:  # the oracle and the bounds on a part of them
        eng = engine(npipes=ni)
        z = np.zeros((n, 3))
        eng.set_j_particles(0.0, m, z, z, v, x)
        eng.set_ti(0.0)
        eng.calc_firsthalf(n, members.astype(np.int32), x[members], v[members], eps2)
        out = eng.calc_lasthalf2()
        eng.close()
        part = np.r_[0:40, ni - 40:ni]
        got, members = tuple(q[part] for q in out), members[part]
    else:
        got = run(m, x, v, members, eps2)
    ref = oracle.force(x, v, m, members.astype(np.int32), x[members], v[members], eps2)
    check(got, ref, bounds(m, x, v, members, eps2))
    assert np.array_equal(got[3], ref[3])


@pytest.mark.parametrize("n", [130, 1030])
def test_index_not_address(oracle, n):
    m, x, v = cluster(n, n)
    index = np.random.default_rng(n).permutation(n).astype(np.int32)
    members = np.arange(0, n, 7)
    got = run(m, x, v, members, 0.0, index=index)
    ref = oracle.force(x, v, m, index[members], x[members], v[members], 0.0, jindex=index)
    check(got, ref, bounds(m, x, v, members, 0.0))
    assert np.array_equal(got[3], ref[3])


# a lattice: six nearest neighbours at one distance in different runs, tiles
# and splits; two interleaved scales, so that r^2 agree in their upper word
# without being equal
@pytest.mark.parametrize("side,jitter", [(4, 0.0), (11, 0.0), (11, 1e-9), (17, 0.0)])
def test_ties(oracle, side, jitter):
    g = np.arange(side, dtype=float)
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(side)
    x = x[rng.permutation(len(x))] + jitter * rng.uniform(-1, 1, (len(x), 3))
    n = len(x)
    m, v = np.full(n, 1.0 / n), rng.normal(size=(n, 3))
    members = np.arange(0, n, max(1, n // 200))
    got = run(m, x, v, members, 0.0)
    ref = oracle.force(x, v, m, members.astype(np.int32), x[members], v[members], 0.0)
    assert np.array_equal(got[3], ref[3])
    check(got, ref, bounds(m, x, v, members, 0.0))


@pytest.mark.parametrize("n,ni", [(50, 2), (300, 20), (700, 64)])
def test_outside_the_normal_range(oracle, n, ni):
    m, x, v = cluster(n, n + 5)
    x[3] = x[1]                        # coincident: pot -inf for both
    x[4] = 0.0
    x[5] = [1e-160, 0.0, 0.0]          # r^2 = 1e-320, subnormal
    x[7] = [1e160, 0.0, 0.0]           # r^2 overflows against every other
    members = np.unique(np.r_[1, 3, 4, 5, 7, np.arange(n - ni, n)])
    got = run(m, x, v, members, 0.0)
    with np.errstate(all="ignore"):
        ref = oracle.force(x, v, m, members.astype(np.int32), x[members], v[members], 0.0)
        tol = bounds(m, x, v, members, 0.0)
    odd = np.isin(members, (1, 3, 4, 5, 7))
    check(got, ref, tol, rows=~odd)
    for k in range(2):  # a force is finite on both sides or on neither
        assert np.array_equal(np.isfinite(got[k]).all(1), np.isfinite(ref[k]).all(1)), k
    # the oracle divides by r^2, which overflows below 2^-1024: the potential
    # of the close pair is its one dominant term
    want = ref[2].copy()
    want[members == 4], want[members == 5] = -m[5] / 1e-160, -m[4] / 1e-160
    rel = 2 * (n + 40) * 2.0 ** -53

    def check_pot(pot):
        ok = np.isfinite(want)
        assert np.array_equal(pot[~ok], want[~ok])
        # r^2 itself, subnormal, carries 2^-1074 of rounding: half of that on 1 / r
        sub = np.isin(members, (4, 5)) * (0.5 * (2.0 ** -1074 / 1e-320))
        assert np.all(np.abs(pot[ok] - want[ok]) <= (rel + sub[ok]) * np.abs(want[ok]))

    check_pot(got[2])
    assert np.array_equal(got[3], ref[3])
    # the same through the potential-only kernel
    eng = engine()
    z = np.zeros((n, 3))
    eng.set_j_particles(0.0, m, z, z, v, x)
    eng.set_ti(0.0)
    check_pot(eng.potential(n, members.astype(np.int32), x[members], 0.0))
    eng.close()
