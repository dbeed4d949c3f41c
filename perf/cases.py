"""What a user of the force engine has it do, as cases that can be timed.

Every case goes through the package's public entry points with host arrays,
as a host program linked against the libraries drives them: single blocks of
a block-timestep integration, whole sweeps, energies, the GRAPE-4 ABI, an
ensemble of clusters, the two force-call servers and the snapshot reader.

Clusters are seeded Plummer spheres in N-body units; the j-state carries the
smooth field's acceleration and jerk, so the prediction to a block time moves
the particles as an integration does.
"""
import math

import numpy as np
import torch

from starlab_b200 import ics
from starlab_b200.ensemble import Ensemble
from starlab_b200.g6 import G6Engine
from starlab_b200.grape4 import H3Engine
from starlab_b200.server import ResidentServer, Server
from starlab_b200.story import StoryReader, format_story

T_BLOCK = 1.0 / 128  # block time of the single calls; the j-state is at time 0
LIST_MAX = 512       # neighbours read back per particle (a few tens are found)
T_LAST = 1.0 / 256   # time of the previous block's corrected particles


def listed():
    return [
        # One block step of kira at N = 1024 (its default size): the previous
        # block's corrected particles go in, the next block's forces come
        # out.  Blocks are small and there are millions of them: latency.
        {"name": "kira_block_1k", "kind": "block", "n": 1024, "ni": 24, "nb_radius": 0.0, "eps2": 1e-6,
         "precision": "fp64", "salpeter": False},
        # The same for an unsoftened cluster of a few ten thousand stars with
        # a mass spectrum, an odd count: kira's usual production size.
        {"name": "kira_block_40k", "kind": "block", "n": 40009, "ni": 61, "nb_radius": 0.0, "eps2": 0.0,
         "precision": "fp64", "salpeter": True},
        # One full chunk of pipelines (256 i) at N = 65536 with neighbour
        # lists of radius 0.05, as kira asks for them around perturbed binaries.
        {"name": "call_lists_64k", "kind": "block", "n": 65536, "ni": 256, "nb_radius": 0.05, "eps2": 1e-6,
         "precision": "fp64", "salpeter": False},
        # A large block of a 262144-body mass-spectrum cluster in the mixed mode.
        {"name": "call_mixed_256k", "kind": "block", "n": 262144, "ni": 4096, "nb_radius": 0.0, "eps2": 1e-8,
         "precision": "mixed", "salpeter": True},
        # Forces on every particle (the start of a run, or a synchronised
        # block), FP64 at N = 65536 ...
        {"name": "sweep_fp64_64k", "kind": "sweep", "n": 65536, "eps2": 1e-6, "precision": "fp64", "salpeter": False},
        # ... and the benchmark's mixed-mode workload, N = 262144.
        {"name": "sweep_mixed_256k", "kind": "sweep", "n": 262144, "eps2": 1e-8, "precision": "mixed",
         "salpeter": True},
        # Energies and potentials of a snapshot (what hsys_stats asks for).
        {"name": "energies_fp64_64k", "kind": "energies", "n": 65536, "eps2": 1e-6, "precision": "fp64",
         "salpeter": True},
        # kira's other hardware branch: the GRAPE-4 ABI, every particle
        # against every other in chunks of its pipeline count.
        {"name": "grape4_sweep_20k", "kind": "grape4", "n": 20011},
        # Many independent clusters integrated together, states read back.
        {"name": "ensemble_64", "kind": "ensemble", "clusters": 64, "n_lo": 256, "n_hi": 16384, "t_end": 1.0 / 32,
         "precision": "mixed"},
        # A burst of force calls of many integrations, batched by the server:
        # block sizes from p(ni) ~ 1/ni as block timesteps give them.
        {"name": "served_burst", "kind": "served", "resident": False, "clusters": 24, "n_lo": 512, "n_hi": 65536,
         "calls": 96, "precision": "mixed"},
        # The same from smaller clusters through the device-resident loop.
        {"name": "resident_burst", "kind": "served", "resident": True, "clusters": 24, "n_lo": 512, "n_hi": 8192,
         "calls": 96, "precision": "mixed"},
        # A snapshot file read from host bytes, corrected as get_dyn does.
        {"name": "story_64k", "kind": "story", "n": 65536, "raw": False, "device": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "block", "block", "sweep", "energies", "grape4", "ensemble", "served", "story"])
    precision = rng.choice(["fp64", "mixed"])
    eps2 = rng.choice([0.0, 1e-8, 1e-6, 1e-4])
    salpeter = rng.random() < 0.5
    if kind == "block":
        n = _log(rng, 600, 262144)
        ni = min(n // 2, _log(rng, 1, 8192 if precision == "mixed" else 4096))
        radius = 0.05 if rng.random() < 0.3 and ni <= 1024 and n <= 65536 else 0.0
        return {"kind": kind, "n": n, "ni": ni, "nb_radius": radius, "eps2": eps2, "precision": precision,
                "salpeter": salpeter}
    if kind in ("sweep", "energies"):
        n = _log(rng, 2000, 200000 if precision == "mixed" else 100000)
        return {"kind": kind, "n": n, "eps2": eps2, "precision": precision, "salpeter": salpeter}
    if kind == "grape4":
        return {"kind": kind, "n": _log(rng, 1000, 60000)}
    if kind == "ensemble":
        return {"kind": kind, "clusters": _log(rng, 8, 128), "n_lo": 128, "n_hi": _log(rng, 1024, 12000),
                "t_end": 1.0 / 64, "precision": precision}
    if kind == "served":
        return {"kind": kind, "resident": rng.random() < 0.5, "clusters": _log(rng, 6, 32), "n_lo": 300,
                "n_hi": _log(rng, 4096, 40000), "calls": _log(rng, 24, 160), "precision": precision}
    return {"kind": kind, "n": _log(rng, 2000, 60000), "raw": rng.random() < 0.5, "device": rng.random() < 0.5}


# ------------------------------------------------------------------ inputs

def _cluster(n, seed, salpeter=False):
    """(m, x, v, a, j): a Plummer sphere and the smooth field's acceleration
    and its rate of change along the orbits."""
    masses = ics.salpeter_masses(n, seed + 1) if salpeter else None
    m, x, v = ics.plummer(n, seed, masses=masses)
    b2 = (3.0 * math.pi / 16.0) ** 2
    s = 1.0 / np.sqrt((x * x).sum(1, keepdims=True) + b2)
    a = -x * s ** 3
    j = -v * s ** 3 + 3.0 * x * (x * v).sum(1, keepdims=True) * s ** 5
    return m, x, v, a, j


def _predict(x, v, a, j, h):
    return x + h * (v + h * (0.5 * a + h * (j / 6.0))), v + h * (a + h * (0.5 * j))


class _Handle:
    """An engine of its own cluster id, closed with the state that holds it."""
    used = 0

    def __init__(self, precision, npipes):
        _Handle.used += 1
        self.eng = G6Engine(cluster_id=_Handle.used, precision=precision, npipes=npipes)

    def __del__(self):
        self.eng.close()


_servers = {}


class _Clusters:
    """Clusters of one of the process's servers, closed with the state."""

    def __init__(self, case, clusters, eps2):
        key = (case["resident"], case["precision"])
        if key not in _servers:
            _servers[key] = (ResidentServer if case["resident"] else Server)(precision=case["precision"])
        self.server, self.ids = _servers[key], []
        for m, x, v, a, j in clusters:
            c = self.server.open_cluster(len(m), eps2)
            self.ids.append(c)
            self.server.set_j(c, 0.0, m, j / 6.0, 0.5 * a, v, x)

    def __del__(self):
        for c in self.ids:
            self.server.close_cluster(c)


SERVED_EPS2 = 1e-6


def _block(case, seed):
    """The cluster, the previous block's corrected particles and the next
    block's members: address lists and states."""
    m, x, v, a, j = _cluster(case["n"], seed, case["salpeter"])
    rng = np.random.default_rng(seed + 2)
    last = np.sort(rng.choice(case["n"], case["ni"], replace=False)).astype(np.int32)
    members = np.sort(rng.choice(case["n"], case["ni"], replace=False)).astype(np.int32)
    xl, vl = _predict(x[last], v[last], a[last], j[last], T_LAST)
    return m, x, v, a, j, last, members, xl, vl


def _spread(count, salt):
    """`count` values evenly spread over [0, 1), jittered, in no order."""
    rng = np.random.default_rng(salt)
    return (rng.permutation(count) + rng.uniform(0.0, 1.0, count)) / count


def _sizes(case):
    """The clusters' sizes, log-uniform: the case's own, the same for every seed."""
    lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
    return np.exp(lo + _spread(case["clusters"], case["n_hi"]) * (hi - lo)).astype(int)


def _call_sizes(case):
    """(cluster, its n, ni) of each call of a burst, ni from p(ni) ~ 1/ni."""
    ns, u = _sizes(case), _spread(case["calls"], case["n_hi"] + 1)
    out = []
    for q in range(case["calls"]):
        n = int(ns[q % len(ns)])
        out.append((q % len(ns), n, min(n, max(1, int(math.exp(u[q] * math.log(n)))))))
    return out


def _served(case, seed):
    clusters = [_cluster(int(n), 1000 * seed + k) for k, n in enumerate(_sizes(case))]
    rng = np.random.default_rng(seed + 3)
    calls = []
    for q, (c, n, ni) in enumerate(_call_sizes(case)):
        i0 = int(rng.integers(0, n - ni + 1))
        ti = 1e-5 * (q + 1)
        _, x, v, a, j = clusters[c]
        xi, vi = _predict(x[i0:i0 + ni], v[i0:i0 + ni], a[i0:i0 + ni], j[i0:i0 + ni], ti)
        calls.append((c, ti, np.arange(i0, i0 + ni, dtype=np.int32), xi, vi))
    return clusters, calls


def prepare(case, seed):
    kind = case["kind"]
    if kind == "block":
        m, x, v, a, j, last, members, xl, vl = _block(case, seed)
        h = _Handle(case["precision"], max(case["ni"], 256))
        h.eng.set_j_particles(0.0, m, j / 6.0, 0.5 * a, v, x)
        xi, vi = _predict(x, v, a, j, T_BLOCK)
        up = np.isin(members, last)
        xi, vi = xi[members], vi[members]
        if up.any():  # members of the previous block too: predicted from their corrected state
            k = np.searchsorted(last, members[up])
            b = members[up]
            xi[up], vi[up] = _predict(xl[k], vl[k], a[b], j[b], T_BLOCK - T_LAST)
        return {"case": case, "h": h, "n": case["n"], "last": last, "tl": np.full(case["ni"], T_LAST), "ml": m[last],
                "jl": j[last] / 6.0, "al": 0.5 * a[last], "vl": vl, "xl": xl, "members": members, "xi": xi, "vi": vi,
                "h2": np.full(case["ni"], case["nb_radius"] ** 2)}
    if kind in ("sweep", "energies"):
        m, x, v, a, j = _cluster(case["n"], seed, case["salpeter"])
        return {"case": case, "h": _Handle(case["precision"], 256), "n": case["n"], "m": m, "x": x, "v": v,
                "a2": 0.5 * a, "j6": j / 6.0}
    if kind == "grape4":
        m, x, v, a, j = _cluster(case["n"], seed)
        return {"case": case, "h3": H3Engine(), "n": case["n"], "m": m, "x": x, "v": v,
                "a2": 0.5 * a, "j6": j / 6.0}
    if kind == "ensemble":
        ns = _sizes(case)
        cl = [ics.plummer(int(n), 1000 * seed + k) for k, n in enumerate(ns)]
        ens = Ensemble([c[0] for c in cl], [c[1] for c in cl], [c[2] for c in cl], (4.0 / ns) ** 2, eta=0.02,
                       precision=case["precision"])
        return {"case": case, "ens": ens}
    if kind == "served":
        clusters, calls = _served(case, seed)
        cl = _Clusters(case, clusters, SERVED_EPS2)
        return {"case": case, "cl": cl, "calls": calls, "n": [len(c[0]) for c in clusters]}
    m, x, v = _snapshot(case, seed)
    text = format_story(m, x, v, log_lines=[" ===>  snapshot"])
    st = {"case": case, "rd": StoryReader(), "text": text}
    if case["device"]:
        st["dev"] = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    return st


def _snapshot(case, seed):
    m, x, v = ics.plummer(case["n"], seed, masses=ics.salpeter_masses(case["n"], seed + 1))
    return m, x + 1e-3, v - 5e-4


# --------------------------------------------------------------------- run

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "block":
        eng = state["h"].eng
        eng.set_j_particles(state["tl"], state["ml"], state["jl"], state["al"], state["vl"], state["xl"],
                            address=state["last"], index=state["last"])
        eng.set_ti(T_BLOCK)
        lists = case["nb_radius"] > 0
        eng.calc_firsthalf(state["n"], state["members"], state["xi"], state["vi"], case["eps2"],
                           state["h2"] if lists else None)
        acc, jerk, pot, nn = eng.calc_lasthalf2()
        if not lists:
            return {"acc": acc, "jerk": jerk, "pot": pot, "nn": nn}
        eng.read_neighbour_list()
        count, rows = np.empty(case["ni"], np.int32), np.full((case["ni"], LIST_MAX), -1, np.int32)
        for p in range(case["ni"]):
            got = eng.get_neighbour_list(p, LIST_MAX)[1]
            count[p], rows[p, :len(got)] = len(got), got
        return {"acc": acc, "jerk": jerk, "pot": pot, "nn": nn, "count": count, "lists": rows}
    if kind in ("sweep", "energies"):
        eng = state["h"].eng
        eng.set_j_particles(0.0, state["m"], state["j6"], state["a2"], state["v"], state["x"])
        eng.set_ti(T_BLOCK)
        if kind == "energies":
            epot, ekin, pot = eng.energies(state["n"], case["eps2"], want_pot=True)
            return {"epot": epot, "ekin": ekin, "pot": pot}
        acc, jerk, pot, nn = eng.sweep(state["n"], eps2=case["eps2"])
        return {"acc": acc, "jerk": jerk, "pot": pot, "nn": nn}
    if kind == "grape4":
        h3, n, x, v = state["h3"], state["n"], state["x"], state["v"]
        # kira's GRAPE-4 branch stores the block itself at the block time
        h3.set_j_particles(x, v, state["a2"], state["j6"], state["m"], T_BLOCK)
        h3.setti(T_BLOCK)
        np_ = h3.npipe()
        got = [h3.calc(n, x[i:i + np_], v[i:i + np_], 0.0, 0.0) for i in range(0, n, np_)]
        return {k: np.concatenate([g[q] for g in got]) for q, k in enumerate(("acc", "jerk", "pot"))}
    if kind == "ensemble":
        ens = state["ens"]
        ens.start()
        ens.run(case["t_end"])
        got = [ens.get(c) for c in range(len(ens.n))]
        return {k: np.concatenate([g[k] for g in got]) for k in ("x", "v", "acc", "jerk", "t", "dt")}
    if kind == "served":
        cl, n = state["cl"], state["n"]
        ids = [cl.server.submit(cl.ids[c], ti, n[c], idx, xi, vi) for c, ti, idx, xi, vi in state["calls"]]
        got = [cl.server.wait(r) for r in ids]
        return {k: np.concatenate([g[q] for g in got]) for q, k in enumerate(("acc", "jerk", "pot", "nn"))}
    rd = state["rd"]
    if case["device"]:
        info = rd.parse_device(state["dev"].data_ptr(), state["dev"].numel(), raw=case["raw"])
        m, x, v = rd.leaves(info)
        return {"mass": m, "pos": x, "vel": v}
    s = rd.parse(state["text"], raw=case["raw"])
    return {"mass": s.leaves_mass, "pos": s.leaves_pos, "vel": s.leaves_vel, "index": s.index, "parent": s.parent,
            "node_mass": s.mass, "node_pos": s.pos, "node_vel": s.vel}


# -------------------------------------------------------------------- work

J_BYTES = 104        # a j-particle as it is sent: t, m, x, v, a/2, j/6
I_BYTES = 52         # an i-particle: x, v, index
OUT_BYTES = 60       # acc, jerk, pot, nn
PAIR_FLOPS = 60      # the customary count of one acc + jerk interaction
POT_FLOPS = 20       # one potential interaction


def work(case):
    kind = case["kind"]
    if kind == "block":
        n, ni = case["n"], case["ni"]
        return {"bytes": J_BYTES * n + (J_BYTES + I_BYTES + OUT_BYTES) * ni, "flops": PAIR_FLOPS * n * ni}
    if kind == "sweep":
        n = case["n"]
        return {"bytes": (J_BYTES + OUT_BYTES) * n, "flops": PAIR_FLOPS * n * n}
    if kind == "energies":
        n = case["n"]
        return {"bytes": (J_BYTES + 8) * n, "flops": POT_FLOPS * n * n}
    if kind == "grape4":
        n = case["n"]
        return {"bytes": (J_BYTES + 48 + 56) * n, "flops": PAIR_FLOPS * n * n}
    if kind == "ensemble":
        # every particle's state in and out, and at least one force on each
        # at t = 0 and at each of the largest steps (1/16 at most) after it
        ns = _sizes(case)
        return {"bytes": int(ns.sum()) * (56 + 14 * 8), "flops": PAIR_FLOPS * 2.0 * float((ns.astype(float) ** 2).sum())}
    if kind == "served":
        calls = _call_sizes(case)
        return {"bytes": sum(J_BYTES * n + (I_BYTES + OUT_BYTES) * ni for _, n, ni in calls),
                "flops": PAIR_FLOPS * sum(n * ni for _, n, ni in calls)}
    return {"bytes": (275 + 56) * case["n"], "flops": 0}


# ------------------------------------------------------------------- exact

def _direct(xi, vi, idx, xj, vj, m, eps2, pot_only=False):
    """Direct sums in 64 bits: (acc, jerk, pot), the particle idx[i] left out."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda q: torch.from_numpy(np.ascontiguousarray(q)).to(dev)  # noqa: E731
    xi, vi, xj, vj, m, idx = t(xi), t(vi), t(xj).T.contiguous(), t(vj).T.contiguous(), t(m), t(idx).long()
    ni, n = xi.shape[0], xj.shape[1]
    acc = torch.zeros(ni, 3, dtype=torch.float64, device=dev)
    jerk, pot = torch.zeros_like(acc), torch.zeros(ni, dtype=torch.float64, device=dev)
    step = max(1, (1 << 25) // n)
    for s in range(0, ni, step):
        e = min(ni, s + step)
        d = [xj[c] - xi[s:e, c, None] for c in range(3)]
        w = d[0] * d[0]
        w.addcmul_(d[1], d[1]).addcmul_(d[2], d[2]).add_(eps2)
        w[torch.arange(e - s, device=dev), idx[s:e]] = math.inf
        w.rsqrt_()
        q = w * m  # m / r
        pot[s:e] = -q.sum(1)
        if pot_only:
            continue
        w.mul_(w)  # 1 / r^2
        q.mul_(w)  # m / r^3
        rv = torch.zeros_like(w)
        for c in range(3):
            dv = vj[c] - vi[s:e, c, None]
            rv.addcmul_(d[c], dv)
            jerk[s:e, c] = dv.mul_(q).sum(1)
            acc[s:e, c] = torch.mul(q, d[c], out=dv).sum(1)
        rv.mul_(w).mul_(q).mul_(-3.0)
        for c in range(3):
            jerk[s:e, c] += d[c].mul_(rv).sum(1)
    return acc.cpu().numpy(), jerk.cpu().numpy(), pot.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "block":
        m, x, v, a, j, last, members, xl, vl = _block(case, seed)
        xj, vj = _predict(x, v, a, j, T_BLOCK)
        xj[last], vj[last] = _predict(xl, vl, a[last], j[last], T_BLOCK - T_LAST)
        acc, jerk, pot = _direct(xj[members], vj[members], members, xj, vj, m, case["eps2"])
        out = {"acc": acc, "jerk": jerk, "pot": pot, "nn": None}
        if case["nb_radius"] > 0:
            out.update(count=None, lists=None)
        return out
    if kind in ("sweep", "energies"):
        m, x, v, a, j = _cluster(case["n"], seed, case["salpeter"])
        x, v = _predict(x, v, a, j, T_BLOCK)
        acc, jerk, pot = _direct(x, v, np.arange(case["n"]), x, v, m, case["eps2"], pot_only=kind == "energies")
        if kind == "energies":
            return {"epot": 0.5 * float((m * pot).sum()), "ekin": 0.5 * float((m * (v * v).sum(1)).sum()), "pot": pot}
        return {"acc": acc, "jerk": jerk, "pot": pot, "nn": None}
    if kind == "grape4":
        m, x, v, _, _ = _cluster(case["n"], seed)
        acc, jerk, pot = _direct(x, v, np.arange(case["n"]), x, v, m, 0.0)
        return {"acc": acc, "jerk": jerk, "pot": pot}
    if kind == "served":
        clusters, calls = _served(case, seed)
        got = []
        for c, ti, idx, xi, vi in calls:
            m, x, v, a, j = clusters[c]
            xj, vj = _predict(x, v, a, j, ti)
            got.append(_direct(xi, vi, idx, xj, vj, m, SERVED_EPS2))
        out = {k: np.concatenate([g[q] for g in got]) for q, k in enumerate(("acc", "jerk", "pot"))}
        return dict(out, nn=None)
    if kind == "story":
        m, x, v = _snapshot(case, seed)
        if case["raw"]:  # 18 digits give the values back
            out = {"mass": m, "pos": x, "vel": v}
        else:  # the root takes the centre of mass, the leaves stay where they are
            out = {"mass": m, "pos": None, "vel": None}
        if not case["device"]:
            out.update(index=None, parent=None, node_mass=None, node_pos=None, node_vel=None)
        return out
    return None  # an integration has no value that is quick to state
