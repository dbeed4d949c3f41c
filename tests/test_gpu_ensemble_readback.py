"""The state read right after a per-cluster run is the run's: it goes back to
the device on the stream that the read-back and the energies run on."""
import numpy as np
import pytest

from starlab_b200 import ics

pytestmark = pytest.mark.gpu


def test_state_after_a_per_cluster_run():
    import torch
    from starlab_b200.ensemble import Ensemble
    sizes = (1, 700, 12000, 33)  # a state of several hundred kB a row, odd tails
    cl = [ics.plummer(n, 900 + n) for n in sizes]
    ens = Ensemble([c[0] for c in cl], [c[1] for c in cl], [c[2] for c in cl], 1e-2)
    for t_end in (2.0 ** -9, 2.0 ** -8):
        if t_end == 2.0 ** -9:
            ens.start()
        ens.run(t_end, per_cluster=True)
        now = [ens.get(c) for c in range(len(sizes))]
        ek, ep = ens.energies()
        torch.cuda.synchronize()
        later = [ens.get(c) for c in range(len(sizes))]
        for c, (a, b) in enumerate(zip(now, later)):
            for k in a:
                assert np.array_equal(a[k], b[k]), (t_end, c, k)
            assert np.all(a["dt"] > 0.0) and np.all(a["t"] == t_end), c  # every step ends on it
            assert np.array_equal(a["m"], cl[c][0])
        k2 = [0.5 * np.sum(a["m"] * np.sum(a["v"] ** 2, 1)) for a in now]
        assert np.allclose(ek, k2, rtol=1e-12)
    ens.close()
