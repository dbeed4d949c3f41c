"""The FP64 kernels with two i per thread (blocks of 8192 i and more): edges of
the 512-i tiles and of the runs of sixteen records, tied neighbours, squared
distances outside the normal range, neighbour lists, and the GRAPE-4 pipeline,
against the oracles.

Tolerance: each side's sum of n terms is within (n + 40) u sum|term| of the
exact one (u = 2^-53; 40 covers a term's own roundings), so the two differ by
at most twice that; the GRAPE-4 pipeline's is the parity tests' 1e-12."""
import os
import subprocess
import sys

import numpy as np
import pytest

from test_gpu_fp64_pairs import bounds, check, cluster

pytestmark = pytest.mark.gpu

_cid = [7800]


def run(m, x, v, ni, eps2, config=None, index=None, h2=None):
    """The first ni particles' forces, and the shape they ran in."""
    from starlab_b200 import G6Engine
    n = len(m)
    _cid[0] += 1
    eng = G6Engine(cluster_id=_cid[0], precision="fp64", npipes=ni)
    z = np.zeros((n, 3))
    eng.set_j_particles(0.0, m, z, z, v, x, index=index)
    eng.set_ti(0.0)
    if config:
        eng.set_config(*config)
    idx = np.arange(ni) if index is None else index[:ni]
    eng.calc_firsthalf(n, idx.astype(np.int32), x[:ni], v[:ni], eps2, h2)
    out, cfg = eng.calc_lasthalf2(), eng.last_config()
    lists = None
    if h2 is not None:
        assert eng.read_neighbour_list() == 0
        lists = [eng.get_neighbour_list(k) for k in (0, ni // 2, ni - 1)]
    eng.close()
    assert cfg[1] == 2, cfg
    return out, lists


def some(ni):
    """A few i of every tile edge, lane and warp."""
    return np.unique(np.clip(np.r_[0:3, 31:34, 63:66, 255:258, 511:514, ni // 2, ni - 34:ni], 0, ni - 1))


@pytest.mark.parametrize("n,ni,config", [
    (10000, 9000, None), (10000, 10000, None),        # the shape the engine takes by itself
    (129, 65, (32, 2, 8, 8, 1)), (1000, 513, (32, 2, 8, 1, 3)), (1025, 512, (32, 2, 8, 2, 9)),
    (2049, 511, (32, 2, 8, 4, 5)), (700, 700, (32, 2, 8, 1, 1))])
@pytest.mark.parametrize("eps2", [0.0, 1e-4])
def test_sizes(oracle, n, ni, config, eps2):
    m, x, v = cluster(n, n + ni)
    got, _ = run(m, x, v, ni, eps2, config)
    k = some(ni)
    ref = oracle.force(x, v, m, k.astype(np.int32), x[k], v[k], eps2)
    check([q[k] for q in got], ref, bounds(m, x, v, k, eps2))
    assert np.array_equal(got[3][k], ref[3])


@pytest.mark.parametrize("config", [(32, 2, 8, 1, 3), (32, 2, 8, 8, 2)])
def test_ties_index_and_lists(oracle, config):
    g = np.arange(11.0)
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(3)
    x = x[rng.permutation(len(x))]
    n = len(x)
    m, v = np.full(n, 1.0 / n), rng.normal(size=(n, 3))
    k = some(600)
    for index in (None, rng.permutation(n).astype(np.int32)):
        got, lists = run(m, x, v, 600, 0.0, config, index, np.full(600, 1.5))
        ids = (np.arange(n) if index is None else index).astype(np.int32)
        ref = oracle.force(x, v, m, ids[k], x[k], v[k], 0.0, jindex=ids)
        assert np.array_equal(got[3][k], ref[3])
        check([q[k] for q in got], ref, bounds(m, x, v, k, 0.0))
        for (rc, q), i in zip(lists, (0, 300, 599)) if index is None else ():
            near = np.flatnonzero(((x - x[i]) ** 2).sum(1) < 1.5)
            assert rc == 0 and set(q.tolist()) - {i} == set(near.tolist()) - {i}


@pytest.mark.parametrize("config", [(32, 2, 8, 1, 2), (32, 2, 8, 8, 3)])
def test_outside_the_normal_range(oracle, config):
    n, ni = 700, 530
    m, x, v = cluster(n, 9)
    x[3], x[4], x[5], x[7] = x[1], 0.0, [1e-160, 0.0, 0.0], [1e160, 0.0, 0.0]
    got, _ = run(m, x, v, ni, 0.0, config)
    k = np.unique(np.r_[some(ni), 1, 3, 4, 5, 7])
    with np.errstate(all="ignore"):
        ref = oracle.force(x, v, m, k.astype(np.int32), x[k], v[k], 0.0)
        tol = bounds(m, x, v, k, 0.0)
    odd = np.isin(k, (1, 3, 4, 5, 7))
    mine = [q[k] for q in got]
    check(mine, ref, tol, rows=~odd)
    for q in range(2):
        assert np.array_equal(np.isfinite(mine[q]).all(1), np.isfinite(ref[q]).all(1))
    assert np.all(np.isneginf(mine[2][np.isin(k, (1, 3))])) and np.array_equal(mine[3], ref[3])


GRAPE4 = """
import numpy as np
from starlab_b200.grape4 import H3Engine
from oracle.oracle import G4Oracle
n, ni = 9000, 8700
rng = np.random.default_rng(4)
x, v, m, z = rng.normal(size=(n, 3)), rng.normal(size=(n, 3)), rng.uniform(0.5, 1.0, n) / n, np.zeros((n, 3))
x[40] = x[8000]  # r^2 = 0 without softening: left out by both
eps2 = np.where(np.arange(ni) % 2, 1e-4, 0.0)
h3 = H3Engine()
h3.set_j_particles(x, v, z, z, m, 0.0)
h3.setti(0.0)
got = h3.calc(n, x[:ni], v[:ni], eps2, np.zeros(ni))
k = np.unique(np.r_[0:3, 31:34, 40, 511:514, 8000, ni - 34:ni])
want = G4Oracle().force(x, v, m, x[k], v[k], eps2[k], np.zeros(len(k)))
for a, b in zip(got, want):
    a = a[k]
    e = np.linalg.norm(np.atleast_2d((a - b).T), axis=0) / np.linalg.norm(np.atleast_2d(b.T), axis=0)
    assert e.max() <= 1e-12, e.max()
print("ok")
"""


def test_grape4_pipeline():
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, H3B200_NPIPES="10000")
    out = subprocess.run([sys.executable, "-c", GRAPE4], capture_output=True, text=True, cwd=repo, timeout=300, env=env)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr
