"""FP64 sums close to the largest double: the pair loop holds them scaled by
sqrt(3) (potential) and its cube (acc, jerk), which must not make a finite
force infinite.  Reference: the direct sum in long doubles.

Tolerance: each side's sum of n terms is within (n + 40) u sum|term| of the
exact one (u = 2^-53; 40 covers a term's own roundings)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_cid = [7700]


def direct(m, x, v, i):
    L = np.longdouble
    d, dv = x.astype(L) - x[i].astype(L), v.astype(L) - v[i].astype(L)
    r2 = (d * d).sum(1)
    r2[i] = 1.0
    w = m.astype(L)
    w[i] = 0.0
    mr3 = w / (r2 * np.sqrt(r2))
    rv = (d * dv).sum(1)
    jt = mr3[:, None] * (dv - 3 * (rv / r2)[:, None] * d)
    return (mr3[:, None] * d), jt, -w / np.sqrt(r2)


# m / r^3 of the close pair, and m / r of the heavy one, as a share of the
# largest double: finite on their own, infinite times 3 sqrt(3) or sqrt(3)
@pytest.mark.parametrize("share", [0.25, 0.7])
@pytest.mark.parametrize("n,ni,config", [(50, 1, None), (50, 3, None), (300, 40, None), (700, 300, None), (700, 600, (32, 2, 8, 1, 2)),
                                         (700, 600, (32, 1, 8, 8, 1))])
def test_close_to_the_largest_double(n, ni, config, share):
    from starlab_b200 import G6Engine
    top = np.finfo(float).max
    rng = np.random.default_rng(n + ni)
    m, x, v = rng.uniform(0.5, 1.0, n) / n, rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    m[0] = m[1]
    r = (m[1] / (share * top)) ** (1 / 3)
    x[0], x[1] = 0.0, [r, 0.0, 0.0]            # a force of 1e205 along x, none along y and z but the others'
    v[0], v[1] = 0.0, [0.0, 1e-3, 0.0]
    heavy = share * top * 1e-3                 # its potential: 1e-3 away from i = 2 of mass zero
    x[3] = x[2] + np.array([1e-3, 0.0, 0.0])
    m[2], m[3] = 0.0, heavy * (x[3, 0] - x[2, 0]) / 1e-3
    for case in ("pair", "heavy"):
        mm = m.copy()
        if case == "pair":
            mm[3] = m[1]
        idx = np.arange(ni, dtype=np.int32)
        _cid[0] += 1
        eng = G6Engine(cluster_id=_cid[0], precision="fp64", npipes=ni)
        z = np.zeros((n, 3))
        eng.set_j_particles(0.0, mm, z, z, v, x)
        eng.set_ti(0.0)
        if config:
            eng.set_config(*config)
        eng.calc_firsthalf(n, idx, x[:ni], v[:ni], 0.0)
        acc, jerk, pot, _ = eng.calc_lasthalf2()
        po = eng.potential(n, idx, x[:ni], 0.0)
        eng.close()
        f = (n + 40) * 2.0 ** -53
        for i in (i for i in ((0, 1) if case == "pair" else (2,)) if i < ni):
            at, jt, pt = direct(mm, x, v, i)
            if case == "pair":
                assert np.all(np.abs(acc[i] - at.sum(0)) <= f * np.sqrt((at * at).sum(1)).sum()), i
                assert np.all(np.abs(jerk[i] - jt.sum(0)) <= 4 * f * np.sqrt((jt * jt).sum(1)).sum()), i
            for q in (pot[i], po[i]):
                assert abs(q - pt.sum()) <= f * np.abs(pt).sum(), (case, i)
