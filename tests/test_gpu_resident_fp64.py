"""The resident loop's FP64 calls, batch after batch into the same record
buffers: the nearest neighbours and the sums that are taken again (a pair of
coincident particles) read records that other CTAs of the running kernel have
just written."""
import numpy as np
import pytest

from helpers import rel_err, rel_err_vec, snapshot

pytestmark = pytest.mark.gpu


def test_every_batch_reads_its_own_records(oracle):
    from starlab_b200.server import ResidentServer
    srv = ResidentServer(precision="fp64")
    n = 5000
    m, x, v, a, j = snapshot(n, 77)
    x[901] = x[4200]  # one place at all times, at rest so that it is exactly
    for q in (v, a, j):  # that however it is predicted: pot -inf for these two
        q[901] = q[4200] = 0.0
    c = srv.open_cluster(n, 0.0)
    srv.set_j(c, 0.0, m, j / 6.0, 0.5 * a, v, x)
    rng = np.random.default_rng(5)
    for k in range(40):
        ti = k / 32
        xp, vp = oracle.predict(ti, 0.0, x, v, 0.5 * a, j / 6.0)
        idx = np.unique(np.r_[901, 4200, rng.choice(n, (1, 7, 40)[k % 3], replace=False)]).astype(np.int32)
        acc, jerk, pot, nn = srv.wait(srv.submit(c, ti, n, idx, xp[idx], vp[idx]))[:4]
        with np.errstate(all="ignore"):
            ra, rj, rp, rn, _ = oracle.force(xp, vp, m, idx, xp[idx], vp[idx], 0.0)
        pair = np.isin(idx, (901, 4200))
        assert np.all(np.isneginf(pot[pair])) and np.all(np.isneginf(rp[pair])), k
        assert np.array_equal(nn, rn), k
        f = ~pair
        if f.any():
            # the parity tests' 1e-12 for the sums, and the nearest pair's term,
            # whose distance has the rounding of the predicted positions: a few
            # 2^-53 |x| on either side, three to four times that in the force
            i = idx[f]
            d = np.sqrt(((xp[i] - xp[rn[f]]) ** 2).sum(1))
            tol = 1e-12 + 16 * 2.0 ** -53 * np.abs(xp[i]).max(1) / d
            assert np.all(rel_err_vec(acc[f], ra[f]) < tol) and np.all(rel_err(pot[f], rp[f]) < tol), k
            assert np.all(rel_err_vec(jerk[f], rj[f]) < tol), k
    srv.close()
