"""The workloads whose speed is followed: what users of this framework run.

Simulated annealing is the main path: single calls through
``b200sa.simulated_annealing`` (host arrays, as the reference's binding), batches
through ``b200sa.Plan`` (device buffers) and Boltzmann-machine gradients through
``b200sa.autograd``.  Steepest descent, rotor-model annealing and path-integral
annealing are the other samplers.  The single calls take host arrays and return
host arrays by their nature, so they are timed whole.

Structures are those of ``b200sa.workloads`` (dense, random regular, cubic
lattice, complete graph) and plain sparse random graphs, whose lists differ in
length.  Every case is made from a seed alone.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dwave-samplers_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import b200sa  # noqa: E402
from b200sa import autograd, greedy, sqa, workloads  # noqa: E402


def listed():
    return [
        # The smallest call: one read of a complete graph of 16 spins, 1000
        # sweeps (the sampler's default number).  Set-up and one warp's latency.
        dict(name="single_read", kind="anneal", graph="complete", n=16, degree=0, reads=1, betas=1000,
             per_beta=1, beta0=0.1, beta1=4.2, proposal="Metropolis", random=False),
        # A dense problem of 100 spins, 1000 reads x 1000 sweeps: the ordinary
        # call, in both update orders.
        dict(name="dense", kind="anneal", graph="dense", n=100, degree=50, reads=1000, betas=1000,
             per_beta=1, beta0=0.1, beta1=4.2, proposal="Metropolis", random=False),
        dict(name="dense_random_order", kind="anneal", graph="dense", n=100, degree=50, reads=1000,
             betas=1000, per_beta=1, beta0=0.1, beta1=4.2, proposal="Metropolis", random=True),
        # Sampling at a fixed temperature from a small complete graph.
        dict(name="fixed_beta_gibbs", kind="anneal", graph="complete", n=16, degree=0, reads=4096,
             betas=1, per_beta=2000, beta0=1.0, beta1=1.0, proposal="Gibbs", random=False),
        # A 3D periodic spin glass of 32^3 spins, schedule cut to 64 of its sweeps.
        dict(name="lattice", kind="anneal", graph="cubic", n=32768, degree=6, reads=256, betas=64,
             per_beta=1, beta0=0.1, beta1=3.0, proposal="Metropolis", random=False),
        # A large sparse problem with lists of different lengths, odd sizes.
        dict(name="large_sparse", kind="anneal", graph="sparse", n=20011, degree=6, reads=1023, betas=48,
             per_beta=1, beta0=0.1, beta1=5.0, proposal="Metropolis", random=False),
        # The uneven batch (random-regular problems of all sizes at once) on
        # device buffers: 32 of its 512 problems, schedules cut to a tenth.
        dict(name="uneven_batch", kind="batch", problems=32, n0=64, n1=4096, d0=3, d1=16, r0=32, r1=1024,
             s0=26, s1=205),
        # One gradient of the log partition function of 16 sparse models:
        # fixed-beta Gibbs sampling forward, sample moments backward.
        dict(name="gradient", kind="gradient", models=16, n0=256, n1=2048, degree=6, reads=256, sweeps=100),
        # Steepest descent from random states.
        dict(name="descent", kind="descent", graph="regular", n=2048, degree=6, samples=8192, sparse=False),
        # Rotor-model annealing: the default proposal on a regular graph, and
        # the transverse-field proposal in random order on an irregular one.
        dict(name="rotor", kind="rotor", graph="regular", n=512, degree=6, samples=4096, betas=64, per_beta=1,
             proposal="MetropolisNonErgodic", random=False),
        dict(name="rotor_transverse", kind="rotor", graph="sparse", n=301, degree=5, samples=1000, betas=48,
             per_beta=1, proposal="MetropolisTF", random=True),
        # Path-integral annealing, single-qubit updates.
        dict(name="path_integral", kind="path", graph="regular", n=512, degree=6, samples=4096, betas=16,
             per_beta=1, chain=1, gamma0=5.0, gamma1=0.05, beta0=0.1, beta1=5.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["anneal", "anneal", "anneal", "anneal", "batch", "gradient", "descent", "rotor", "rotor",
                       "path", "path"])
    if kind == "anneal":
        graph = rng.choice(["complete", "dense", "sparse", "regular", "cubic"])
        if graph in ("complete", "dense"):
            n = _log(rng, 5, 300)
            degree = 0 if graph == "complete" else max(2, n // 2)
        elif graph == "cubic":
            n = rng.randrange(4, 33) ** 3
            degree = 6
        else:
            n = _log(rng, 40, 20000)
            degree = rng.randrange(3, 17)
        random = rng.random() < 0.3
        per_read = 10 ** rng.uniform(3.5, 5.3 if random else 5.8)  # attempts of one read
        sweeps = max(1, int(per_read / n))
        reads = max(1, min(_log(rng, 1, 4097), int(2e8 / (sweeps * n))))
        fixed = rng.random() < 0.3
        return dict(kind="anneal", graph=graph, n=n, degree=degree, reads=reads,
                    betas=1 if fixed else sweeps, per_beta=sweeps if fixed else 1,
                    beta0=1.0 if fixed else 0.1, beta1=1.0 if fixed else rng.uniform(2.0, 6.0),
                    proposal=rng.choice(["Metropolis", "Metropolis", "Gibbs"]), random=random)
    if kind == "batch":
        n1 = _log(rng, 300, 4097)
        return dict(kind="batch", problems=rng.randrange(2, 25), n0=rng.randrange(16, 130), n1=n1,
                    d0=3, d1=rng.randrange(4, 17), r0=rng.randrange(1, 64), r1=rng.randrange(64, 1025),
                    s0=rng.randrange(8, 30), s1=rng.randrange(30, 160))
    if kind == "gradient":
        return dict(kind="gradient", models=rng.randrange(1, 17), n0=rng.randrange(64, 300),
                    n1=rng.randrange(300, 2049), degree=rng.randrange(3, 8), reads=_log(rng, 17, 257),
                    sweeps=rng.randrange(10, 101))
    if kind == "descent":
        n = _log(rng, 30, 6000)
        return dict(kind="descent", graph=rng.choice(["regular", "sparse", "dense"]) if n < 300
                    else rng.choice(["regular", "sparse"]),
                    n=n, degree=max(2, n // 2) if n < 40 else rng.randrange(3, 13),
                    samples=max(1, min(_log(rng, 1, 16385), int(1.6e7 / n))), sparse=rng.random() < 0.3)
    if kind == "rotor":
        n = _log(rng, 9, 3000)
        sweeps = max(1, min(rng.randrange(8, 129), 30000 // n))
        return dict(kind="rotor", graph=rng.choice(["regular", "sparse"]), n=n, degree=rng.randrange(3, 9),
                    samples=max(1, min(_log(rng, 1, 8193), int(6e7 / (n * sweeps)))), betas=sweeps, per_beta=1,
                    proposal=rng.choice(list(sqa.PROPOSALS)), random=rng.random() < 0.4)
    n = _log(rng, 12, 1000)
    steps = max(1, min(rng.randrange(4, 33), 8000 // n))
    chain = rng.choice([1, 1, 2, 4])
    return dict(kind="path", graph="regular" if chain == 1 else "chains", n=n - n % chain, degree=rng.randrange(3, 7),
                samples=max(1, min(_log(rng, 1, 16385), int(2.4e7 / (n * steps)))), betas=steps, per_beta=1,
                chain=chain, gamma0=rng.uniform(1.0, 6.0), gamma1=0.05, beta0=0.1, beta1=rng.uniform(1.0, 5.0))


# ---- inputs ------------------------------------------------------------------
def _pairs(n, degree, rng):
    """About n * degree / 2 distinct random pairs u < v, in lexicographic order."""
    m = max(1, n * degree // 2)
    a = rng.integers(0, n, size=int(1.1 * m) + 8)
    b = rng.integers(0, n, size=a.shape[0])
    key = np.unique(np.minimum(a, b)[a != b] * np.int64(n) + np.maximum(a, b)[a != b])
    if key.shape[0] > m:
        key = np.sort(rng.choice(key, m, replace=False))
    return (key // n).astype(np.int32), (key % n).astype(np.int32)


def _graph(case, rng):
    """(n, u, v, J) of the case's structure, couplings of its usual distribution."""
    kind, n = case["graph"], case["n"]
    if kind == "complete":
        u, v = (x.astype(np.int32) for x in np.triu_indices(n, k=1))
        return n, u, v, rng.normal(0.0, 0.3, u.shape[0])
    if kind == "dense":
        u, v = np.triu_indices(n, k=1)
        keep = rng.random(u.shape[0]) < case["degree"] / max(n - 1, 1)
        u, v = u[keep].astype(np.int32), v[keep].astype(np.int32)
        return n, u, v, rng.uniform(-1.0, 1.0, u.shape[0])
    if kind == "cubic":
        inst = workloads.cubic_lattice(L=int(round(n ** (1 / 3))), reads=1, sweeps=1, seed=int(rng.integers(2**31)))
        return n, inst.u, inst.v, inst.J
    if kind == "regular":
        n, u, v = workloads.random_regular(n, case["degree"], rng, int(rng.integers(2**31)))
        return n, u, v, rng.normal(0.0, 1.0, u.shape[0])
    u, v = _pairs(n, case["degree"], rng)
    J = rng.normal(0.0, 1.0, u.shape[0])
    if kind == "chains":  # ferromagnetic chains of consecutive variables
        q = case["chain"]
        inside = (u // q) == (v // q)
        u, v, J = u[~inside], v[~inside], J[~inside]
        k = np.arange(n - 1)
        k = k[k % q != q - 1]
        u = np.concatenate([u, k]).astype(np.int32)
        v = np.concatenate([v, k + 1]).astype(np.int32)
        J = np.concatenate([J, np.full(k.shape[0], -1.8)])
    return n, u, v, J


def _problem(case, seed):
    rng = np.random.default_rng(seed)
    n, u, v, J = _graph(case, rng)
    h = np.zeros(n) if case["graph"] == "cubic" else rng.normal(0.0, 0.1, n)
    return rng, n, u, v, J, h


def _anneal_inputs(case, seed):
    rng, n, u, v, J, h = _problem(case, seed)
    betas = np.geomspace(case["beta0"], case["beta1"], case["betas"])
    if case["graph"] == "cubic":
        betas = np.linspace(case["beta0"], case["beta1"], case["betas"])
    return dict(h=h, u=u, v=v, J=J, betas=betas, states=workloads.random_states(rng, case["reads"], n),
                seed=int(rng.integers(1, 2**40)))


def _descent_inputs(case, seed):
    rng, n, u, v, J, h = _problem(case, seed)
    return dict(h=h, u=u, v=v, J=J, states=workloads.random_states(rng, case["samples"], n))


def _batch_inputs(case, seed):
    """Random-regular problems as in the uneven batch.  The sizes belong to
    the case, graphs, weights and states to the seed."""
    size = np.random.default_rng(case["problems"] + case["n1"])
    rng = np.random.default_rng(seed)
    out = []
    for p in range(case["problems"]):
        n, d, reads, sweeps = (int(size.integers(case[a], case[b] + 1))
                               for a, b in (("n0", "n1"), ("d0", "d1"), ("r0", "r1"), ("s0", "s1")))
        n, u, v = workloads.random_regular(n, d, rng, int(rng.integers(2**31)))
        out.append(workloads.Instance(
            rng.normal(0.0, 0.1, n), u, v, rng.normal(0.0, 1.0, u.shape[0]),
            workloads.random_states(rng, reads, n), np.geomspace(0.1, 5.0, sweeps), 1,
            b200sa.per_read_seeds(1 + 1000003 * seed + 4096 * p, reads)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "anneal":
        return dict(kind=kind, case=case, **_anneal_inputs(case, seed))
    if kind == "descent":
        return dict(kind=kind, case=case, **_descent_inputs(case, seed))
    if kind == "batch":
        insts = _batch_inputs(case, seed)
        plan = b200sa.Plan(insts)
        sin = torch.from_numpy(np.concatenate([p.states.ravel() for p in insts])).cuda()
        return dict(kind=kind, plan=plan, sin=sin, sout=torch.empty_like(sin),
                    en=torch.empty(plan.total_reads, dtype=torch.float64, device="cuda"))
    if kind == "gradient":
        size = np.random.default_rng(case["models"] + case["n1"])
        rng = np.random.default_rng(seed)
        models, hs, Js = [], [], []
        for _ in range(case["models"]):
            n, u, v = workloads.random_regular(int(size.integers(case["n0"], case["n1"] + 1)), case["degree"], rng,
                                               int(rng.integers(2**31)))
            models.append(autograd.IsingModel(n, u, v))
            hs.append(rng.normal(0.0, 0.1, n))
            Js.append(rng.normal(0.0, 0.5, u.shape[0]))
        spec = autograd.SamplingSpec(models, beta=1.0, sweeps=case["sweeps"], reads=case["reads"], seed=seed + 1,
                                     init_seed=seed + 2)
        cat = lambda xs: torch.from_numpy(np.concatenate(xs)).cuda().requires_grad_(True)
        return dict(kind=kind, spec=spec, h=cat(hs), J=cat(Js))
    rng, n, u, v, J, h = _problem(case, seed)
    st = dict(kind=kind, case=case, h=h, u=u, v=v, J=J, seed=int(rng.integers(1, 2**31)))
    if kind == "rotor":
        # Problem field up, transverse field down, in inverse-temperature units.
        st["hp"] = np.geomspace(0.1, 5.0, case["betas"])
        st["hd"] = st["hp"] * np.linspace(1.2, 0.02, case["betas"])
        st["tf"] = rng.uniform(0.5, 1.5, n)
        st["states"] = rng.integers(0, 256, size=(case["samples"], n), dtype=np.uint8)
        return st
    st["hp"] = np.geomspace(case["beta0"], case["beta1"], case["betas"])
    st["hd"] = np.geomspace(case["gamma0"], case["gamma1"], case["betas"])
    st["states"] = workloads.random_states(rng, case["samples"], n)
    st["num_breaks"] = np.zeros((case["samples"], n), dtype=np.intc)
    st["no_breaks"] = np.zeros(0, dtype=np.intc)
    return st


def run(s):
    kind = s["kind"]
    if kind == "batch":
        s["plan"].run(s["sin"], s["sout"], s["en"], stream=torch.cuda.current_stream(), sync=False)
        return s["sout"], s["en"]
    if kind == "gradient":
        return torch.autograd.grad(autograd.log_partition(s["h"], s["J"], s["spec"]), (s["h"], s["J"]))
    c = s["case"]
    states = s["states"].copy()  # annealed in place
    if kind == "anneal":
        return b200sa.simulated_annealing(c["reads"], s["h"], s["u"], s["v"], s["J"], c["per_beta"], s["betas"],
                                          s["seed"], states, c["random"], c["proposal"])
    if kind == "descent":
        return greedy.steepest_gradient_descent(c["samples"], s["h"], s["u"], s["v"], s["J"], states, c["sparse"])
    if kind == "rotor":
        return sqa.simulated_annealing(c["samples"], s["h"], s["u"], s["v"], s["J"], s["tf"], c["per_beta"],
                                       s["hp"], s["hd"], s["seed"], states, c["random"], c["proposal"], 0)[:2]
    out = sqa.path_annealing(c["samples"], s["h"], s["u"], s["v"], s["J"], c["per_beta"], s["hp"], s["hd"], 1.0,
                             -1.8 if c["chain"] > 1 else 0.0, c["chain"], c["chain"], s["seed"], states, 1, 1,
                             s["num_breaks"], s["no_breaks"], s["no_breaks"], 0)
    return out[:2]


def work(case):
    """Bytes: problem, initial states, results, once each.  Operations: two
    per attempted update (scale and compare the delta energy) and two per
    neighbour of it for the samplers that add the local field up each time;
    what a flip adds depends on the data and is left out."""
    kind = case["kind"]
    if kind == "batch":
        n, r, s = ((case[a] + case[b]) / 2 for a, b in (("n0", "n1"), ("r0", "r1"), ("s0", "s1")))
        deg = (case["d0"] + case["d1"]) / 2
        k, updates, row = case["problems"], r * s * n, r * (2 * n + 8)
    elif kind == "gradient":
        n, deg, r = (case["n0"] + case["n1"]) / 2, case["degree"], case["reads"]
        k, updates, row = case["models"], r * case["sweeps"] * n, 8 * n * (1 + deg / 2)
    else:
        n = case["n"]
        deg = n - 1 if case["graph"] == "complete" else case["degree"]
        k, r = 1, case.get("reads", case.get("samples"))
        updates = r * n * case.get("betas", 1) * case.get("per_beta", 1)
        row = r * (2 * n + 8)
    field = kind == "path" or (kind == "rotor" and "NonErgodic" not in case["proposal"])
    return {"bytes": float(k * (row + n * (8 + 8 * deg))),
            "flops": float(k * updates * (2 + (2 * deg if field else 0)))}


# ---- values in 64 bits ---------------------------------------------------------
def exact(case, seed):
    """Energies in 64 bits from plain torch or Python.  The samples themselves
    are whole numbers.  Annealing runs that are long for plain Python have
    none: their energies belong to the states that a run draws."""
    if case["kind"] == "descent" and case["samples"] * case["n"] <= 1 << 25:
        return [None, _descend(_descent_inputs(case, seed)), None]
    if case["kind"] == "anneal" and case["reads"] * case["n"] * case["betas"] * case["per_beta"] <= 300000:
        return [None, _anneal(case, _anneal_inputs(case, seed))]
    return None


def _energy(h, u, v, J, s):
    return float(np.dot(h, s) + np.dot(J, s[u] * s[v]))


def _descend(x):
    """Flip the variable of the least flip energy until none is negative."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = x["h"].shape[0]
    h, J = (torch.from_numpy(x[k]).to(dev) for k in ("h", "J"))
    u, v = (torch.from_numpy(x[k].astype(np.int64)).to(dev) for k in ("u", "v"))
    s = torch.from_numpy(x["states"]).to(dev).double()
    # Neighbour table padded with the extra variable n (coupling zero).
    a, b, w = torch.cat([u, v]), torch.cat([v, u]), torch.cat([J, J])
    order = torch.argsort(a, stable=True)
    a, b, w = a[order], b[order], w[order]
    deg = torch.bincount(a, minlength=n)
    pos = torch.arange(a.shape[0], device=dev) - (torch.cumsum(deg, 0) - deg)[a]
    width = max(int(deg.max()), 1)
    nb = torch.full((n, width), n, dtype=torch.int64, device=dev)
    wt = torch.zeros((n, width), dtype=torch.float64, device=dev)
    nb[a, pos], wt[a, pos] = b, w
    spins = torch.cat([s, torch.zeros(s.shape[0], 1, dtype=torch.float64, device=dev)], dim=1)
    fe = torch.cat([torch.zeros_like(s), torch.full((s.shape[0], 1), math.inf, dtype=torch.float64, device=dev)], 1)
    for i in range(n):
        fe[:, i] = -2 * s[:, i] * (h[i] + spins[:, nb[i]] @ wt[i])
    rows = torch.arange(s.shape[0], device=dev)
    for step in range(1000 * n):
        least, at = fe.min(dim=1)
        go = least < 0
        if step % 16 == 0 and not bool(go.any()):
            break
        su = spins[rows, at]
        fe[rows, at] = torch.where(go, -least, least)
        spins[rows, at] = torch.where(go, -su, su)
        near = nb[at]
        fe.scatter_add_(1, near, go[:, None] * (4 * su)[:, None] * wt[at] * spins.gather(1, near))
        fe[:, n] = math.inf
    s = spins[:, :n]
    return (s @ h + (s[:, u] * s[:, v]) @ J).cpu().numpy()


def _anneal(case, x):
    """One plain Python anneal per read, xorshift128+ numbers."""
    n, mask = x["h"].shape[0], (1 << 64) - 1
    lists = [[] for _ in range(n)]
    for a, b, w in zip(x["u"].tolist(), x["v"].tolist(), x["J"].tolist()):
        lists[a].append((b, w))
        lists[b].append((a, w))
    gibbs = case["proposal"] == "Gibbs"
    energies = []
    for r in range(case["reads"]):
        s = x["states"][r].astype(int).tolist()
        s0, s1 = ((x["seed"] + r) & mask) or mask, 0

        def rand():
            nonlocal s0, s1
            a, b = s0, s1
            a ^= (a << 23) & mask
            s0, s1 = b, a ^ b ^ (a >> 17) ^ (b >> 26)
            return (s1 + b) & mask

        de = [-2 * s[i] * (x["h"][i] + sum(s[j] * w for j, w in lists[i])) for i in range(n)]
        for beta in x["betas"].tolist():
            for _ in range(case["per_beta"]):
                for i in range(n):
                    k = rand() % n if case["random"] else i
                    d = de[k]
                    if d >= 44.36142 / beta:
                        continue
                    if gibbs:
                        flip = float(mask) > float(rand()) * (1.0 + math.exp(d * beta))
                    else:
                        flip = d <= 0.0 or math.exp(-d * beta) * float(mask) > float(rand())
                    if flip:
                        for j, w in lists[k]:
                            de[j] += 4 * s[k] * w * s[j]
                        s[k], de[k] = -s[k], -d
        energies.append(_energy(x["h"], x["u"], x["v"], x["J"], np.array(s, dtype=float)))
    return np.array(energies)
