"""Nearest neighbours of the mixed mode's kernel, which keeps a minimum per
run of records and looks the run through at the end: tied distances in one
run, in different runs, tiles and splits, at sizes around the runs and
tiles, in every lane shape.  Lattice positions are exact on the fixed-point
grid and their squared distances exact in FP32, so the index must be the
oracle's (the first of the tied ones)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_cid = [7400]


@pytest.mark.parametrize("n,ni", [(2, 2), (16, 1), (17, 9), (255, 2), (256, 33), (257, 8), (513, 257), (1331, 600),
                                  (4100, 64)])
def test_ties(oracle, monkeypatch, n, ni):
    from starlab_b200 import G6Engine
    monkeypatch.setenv("G6B200_MIXED_MIN_WORK", "0")  # these sizes would run in FP64 otherwise
    _cid[0] += 1
    eng = G6Engine(cluster_id=_cid[0], precision="mixed", npipes=ni)
    side = int(np.ceil(n ** (1 / 3))) + 1
    g = np.arange(side, dtype=float)
    rng = np.random.default_rng(n)
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    x = np.ascontiguousarray(x[rng.permutation(len(x))[:n]])
    m, v, z = np.full(n, 1.0 / n), rng.normal(size=(n, 3)), np.zeros((n, 3))
    members = np.sort(rng.choice(n, ni, replace=False)).astype(np.int32)
    eng.set_j_particles(0.0, m, z, z, v, x)
    eng.set_ti(0.0)
    eng.calc_firsthalf(n, members, x[members], v[members], 0.0)
    nn = eng.calc_lasthalf2()[3]
    eng.close()
    assert np.array_equal(nn, oracle.force(x, v, m, members, x[members], v[members], 0.0)[3])
