"""Timed cases: the calls a user of this package makes, smallest to largest.

Each case is one call (or one step of a loop) through a public entry point:
`Solver` with host arrays, `PTBatch` for prepared batches, `RBM_PySA` for
device-resident problems, the annealed-importance calls, and the learned
proposal loop.  Sizes are those of the benchmark workloads and the tests, or
generic ones; `draw` spreads over the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pysa_gb300 import Instance, PTBatch, Solver, pack_spins
from pysa_gb300.engine import run_ais_batch
from pysa_gb300.proposal import LearnedProposal, run_with_proposals
from pysa_gb300.rbm import RBM_PySA
from pysa_gb300.utils import lattice_adjacency


def listed():
    return [
        # the smallest call: Solver's defaults (random order, 4 replicas, one
        # read, T = 0.3 .. 1.5) on a small integer Ising problem; launches
        # and latency are what it costs
        dict(name="solver_defaults", kind="solver", ptype="ising",
             values="pm1", n=24, replicas=4, reads=1, sweeps=200, tmin=0.3,
             tmax=1.5, update="random", partition=False),
        # log-partition function from the ladder (get_part_fun), the
        # reference's second headline use
        dict(name="solver_partition", kind="solver", ptype="qubo",
             values="int", n=60, replicas=32, reads=20, sweeps=200, tmin=2.0,
             tmax=40.0, update="sequential", partition=True),
        # the benchmark's dense SK workload, end to end with host arrays:
        # real couplings
        dict(name="solver_sk128", kind="solver", ptype="ising",
             values="normal", n=128, replicas=32, reads=100, sweeps=1000,
             tmin=1.0, tmax=3.5, update="sequential", partition=False),
        # the headline workload: dense integer QUBO, sequential order
        dict(name="batch_qubo1024", kind="batch", ptype="qubo", values="int",
             n=1024, replicas=64, reads=256, sweeps=500, tmin=0.5, tmax=8.0,
             update="sequential"),
        # the same in random order (Solver's default order)
        dict(name="batch_qubo1024_random", kind="batch", ptype="qubo",
             values="int", n=1024, replicas=64, reads=256, sweeps=64,
             tmin=0.5, tmax=8.0, update="random"),
        # planted Wishart: real couplings at the widest tensor-core size
        dict(name="batch_wishart2048", kind="batch", ptype="ising",
             values="wishart", n=2048, replicas=64, reads=128, sweeps=24,
             tmin=0.02, tmax=2.0, update="sequential"),
        # many SK instances of uneven (odd) sizes in one batch
        dict(name="uneven_sk", kind="uneven", ptype="ising", instances=40,
             nmin=64, nmax=1536, replicas=32, reads=100, sweeps=8, tmin=1.0,
             tmax=3.5, update="sequential"),
        # sparse rows: the tutorial's 2-D lattice at the benchmark's size
        dict(name="lattice64", kind="lattice", side=64, replicas=40,
             reads=100, sweeps=50, tmin=1.0, tmax=3.5, update="sequential"),
        # RBM negative phase at the MNIST tutorial's sizes: new couplings
        # every step, everything on the device
        dict(name="rbm_mnist", kind="rbm", visible=784, hidden=128,
             state_size=100, steps=1, tmin=1.0, tmax=1.0),
        # annealed importance sampling of many small instances in one launch
        dict(name="ais_batch24", kind="ais_batch", instances=64, n=24,
             samples=1024, temps=200, beta=2.0, update="sequential"),
        # one annealed_importance call on a wider problem, random order
        # (the entry point's default)
        dict(name="ais_solver96", kind="ais", ptype="ising", n=96,
             samples=1000, temps=200, beta=0.125, reference="uniform",
             update="random"),
        # parallel tempering with the learned proposal: sweeps, online
        # training steps (forward, backward, Adam) and proposal rounds
        dict(name="learned512", kind="learned", instances=32, n=512,
             replicas=64, reads=32, hidden=1024, sweeps=20, tmin=0.3,
             tmax=3.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solver", "partition", "sk", "qubo", "qubo", "wishart",
                       "uneven", "lattice", "rbm", "ais_batch", "ais",
                       "learned"])
    order = rng.choice(["sequential", "random"])
    if kind == "solver":
        return dict(kind="solver", ptype=rng.choice(["ising", "qubo"]),
                    values=rng.choice(["pm1", "int", "normal"]),
                    n=_log_int(rng, 8, 256), replicas=rng.randint(2, 16),
                    reads=rng.randint(1, 8), sweeps=_log_int(rng, 20, 500),
                    tmin=0.3, tmax=1.5, update=order, partition=False)
    if kind == "partition":
        return dict(kind="solver", ptype=rng.choice(["ising", "qubo"]),
                    values="int", n=_log_int(rng, 12, 128),
                    replicas=rng.randint(4, 40), reads=_log_int(rng, 2, 40),
                    sweeps=_log_int(rng, 50, 300), tmin=2.0, tmax=40.0,
                    update=order, partition=True)
    if kind == "sk":
        return dict(kind="solver", ptype="ising", values="normal",
                    n=rng.randint(64, 512), replicas=rng.choice([8, 16, 32]),
                    reads=_log_int(rng, 16, 128),
                    sweeps=_log_int(rng, 100, 500), tmin=1.0, tmax=3.5,
                    update="sequential", partition=False)
    if kind == "qubo":
        return dict(kind="batch", ptype=rng.choice(["ising", "qubo"]),
                    values="int", n=_log_int(rng, 96, 1024),
                    replicas=rng.choice([8, 16, 24, 32, 64]),
                    reads=_log_int(rng, 16, 256),
                    sweeps=_log_int(rng, 16, 64), tmin=0.5, tmax=8.0,
                    update=order)
    if kind == "wishart":
        return dict(kind="batch", ptype="ising", values="wishart",
                    n=rng.randint(700, 2048), replicas=rng.choice([16, 32, 64]),
                    reads=_log_int(rng, 16, 128), sweeps=rng.randint(4, 24),
                    tmin=0.02, tmax=2.0, update="sequential")
    if kind == "uneven":
        return dict(kind="uneven", ptype="ising",
                    instances=_log_int(rng, 8, 40), nmin=rng.randint(16, 200),
                    nmax=_log_int(rng, 300, 1536),
                    replicas=rng.choice([16, 32]), reads=_log_int(rng, 20, 100),
                    sweeps=rng.randint(2, 8), tmin=1.0, tmax=3.5, update=order)
    if kind == "lattice":
        return dict(kind="lattice", side=_log_int(rng, 8, 64),
                    replicas=rng.randint(4, 40), reads=_log_int(rng, 4, 100),
                    sweeps=_log_int(rng, 10, 50), tmin=1.0, tmax=3.5,
                    update=order)
    if kind == "rbm":
        return dict(kind="rbm", visible=_log_int(rng, 36, 784),
                    hidden=_log_int(rng, 16, 256),
                    state_size=_log_int(rng, 10, 100),
                    steps=rng.randint(1, 4), tmin=1.0,
                    tmax=rng.choice([1.0, 3.5]))
    if kind == "ais_batch":
        return dict(kind="ais_batch", instances=_log_int(rng, 4, 64),
                    n=rng.randint(6, 32), samples=_log_int(rng, 64, 1024),
                    temps=_log_int(rng, 50, 200), beta=2.0, update=order)
    if kind == "ais":
        return dict(kind="ais", ptype=rng.choice(["ising", "qubo"]),
                    n=_log_int(rng, 24, 256), samples=_log_int(rng, 100, 1000),
                    temps=_log_int(rng, 50, 200), beta=0.125,
                    reference=rng.choice(["uniform", "uniform", "bernoulli"]),
                    update=order)
    return dict(kind="learned", instances=_log_int(rng, 4, 32),
                n=rng.randint(96, 512), replicas=rng.choice([32, 64]),
                reads=_log_int(rng, 8, 32), hidden=rng.choice([256, 512, 1024]),
                sweeps=20, tmin=0.3, tmax=3.0)


# ------------------------------------------------------------------ problems
def _matrix(values, n, gen):
    """Symmetric [n, n] float32 problem (fields on the diagonal), made on the
    GPU from its generator."""
    dev = gen.device
    if values == "wishart":  # planted: every w orthogonal to the state t
        m = n // 2
        t = 2.0 * torch.randint(0, 2, (n,), generator=gen, device=dev) - 1.0
        w = torch.randn(m, n, generator=gen, device=dev)
        w -= torch.outer(w @ t / n, t)
        J = (w.T @ w) / n
        J = torch.triu(J, 1)
        return (J + J.T).float()
    if values == "normal":
        J = torch.triu(torch.randn(n, n, generator=gen, device=dev), 1)
        return ((J + J.T) / math.sqrt(n)).float()
    if values == "pm1":
        J = 2.0 * torch.randint(0, 2, (n, n), generator=gen, device=dev) - 1.0
        J = torch.triu(J, 1)
        return (J + J.T).float()
    J = torch.randint(-8, 9, (n, n), generator=gen, device=dev).float()
    J = torch.triu(J, 1)
    J = J + J.T
    d = torch.randint(-16, 17, (n,), generator=gen, device=dev).float()
    return J + torch.diag(d)


def _split(P):
    h = np.diag(P).copy()
    J = P.copy()
    np.fill_diagonal(J, 0.0)
    return J, h


def _geometric(case):
    """Inverse temperatures, coldest first, as Solver spaces them."""
    R = case["replicas"]
    ratio = (case["tmax"] / case["tmin"]) ** (1 / max(R - 1, 1))
    return np.array([1 / (case["tmin"] * ratio**k) for k in range(R)],
                    np.float32)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _random_words(batch, gen):
    """Random bit-packed states of every chain (host words; bits past an
    instance's n are zero)."""
    out = np.zeros((batch.num_chains, batch.words), np.uint32)
    for i in range(len(batch.instances)):
        n, c = int(batch.n[i]), int(batch.R[i]) * int(batch.Rd[i])
        x = torch.randint(0, 2, (c, n), generator=gen, device=gen.device,
                          dtype=torch.uint8).cpu().numpy()
        c0 = int(batch.chain_off[i])
        out[c0:c0 + c] = pack_spins(x, "qubo", batch.words)
    return out


# ------------------------------------------------------------------- prepare
def prepare(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    st = {"case": case, "seed": seed}
    if kind == "solver":
        P = _matrix(case["values"], case["n"], gen).cpu().numpy()
        st["solver"] = Solver(P, case["ptype"], "float32")
    elif kind == "batch":
        J, h = _split(_matrix(case["values"], case["n"], gen).cpu().numpy())
        st["batch"] = PTBatch(case["ptype"], [
            Instance(J, h, _geometric(case), case["reads"])])
    elif kind == "uneven":
        # sizes spread evenly over the range, odd ones among them
        I = case["instances"]
        insts = []
        for i in range(I):
            n = case["nmin"] + (case["nmax"] - case["nmin"]) * i // max(I - 1, 1)
            J = _matrix("normal", n, gen).cpu().numpy()
            insts.append(Instance(J, np.zeros(n, np.float32),
                                  _geometric(case), case["reads"]))
        st["batch"] = PTBatch(case["ptype"], insts)
    elif kind == "lattice":
        J = -lattice_adjacency(case["side"], case["side"],
                               sparse=True).astype(np.float32)
        n = case["side"] ** 2
        h = torch.randint(-1, 2, (n,), generator=gen,
                          device=gen.device).float().cpu().numpy()
        st["batch"] = PTBatch("ising", [
            Instance(J, h, _geometric(case), case["reads"])], sparse=True)
    elif kind == "rbm":
        m = RBM_PySA(case["visible"], case["hidden"],
                     state_size=case["state_size"], steps=case["steps"],
                     min_temp=case["tmin"], max_temp=case["tmax"],
                     parallel=False, seed=seed)
        with torch.no_grad():
            for p, s in ((m.W, 1.0), (m.v_bias, 0.5), (m.h_bias, 0.5)):
                p.copy_(s * torch.randn(*p.shape, generator=gen, device="cuda"))
        m.v_state = torch.randint(
            0, 2, m.v_state.shape, generator=gen, device="cuda").float()
        m.h_state = torch.randint(
            0, 2, m.h_state.shape, generator=gen, device="cuda").float()
        st["rbm"] = m
    elif kind == "ais_batch":
        n = case["n"]
        st["instances"] = []
        for _ in range(case["instances"]):
            J = _matrix("normal", n, gen).cpu().numpy()
            x0 = 2.0 * torch.randint(0, 2, (case["samples"], n), generator=gen,
                                     device="cuda").float() - 1.0
            st["instances"].append((np.float32(case["beta"]) * J,
                                    np.zeros(n, np.float32),
                                    x0.cpu().numpy()))
        st["temps"] = (np.arange(1, case["temps"] + 1, dtype=np.float64) /
                       case["temps"]).astype(np.float32)
    elif kind == "ais":
        P = _matrix("pm1", case["n"], gen).cpu().numpy()
        st["solver"] = Solver(P, case["ptype"], "float32")
    elif kind == "learned":
        insts = []
        for _ in range(case["instances"]):
            J = _matrix("pm1", case["n"], gen).cpu().numpy()
            insts.append(Instance(J, np.zeros(case["n"], np.float32),
                                  _geometric(case), case["reads"]))
        b = PTBatch("ising", insts, kernel="tc")
        st["batch"] = b
        st["prop"] = LearnedProposal(b, hidden=case["hidden"], lr=1e-3,
                                     init_seed=seed, target_flips=2.0)
    else:
        raise ValueError(f"unknown kind {kind!r}")
    if "batch" in st:
        st["words"] = _random_words(st["batch"], gen)
    return st


# ----------------------------------------------------------------------- run
_COLUMNS = ("states", "energies", "best_state", "best_energy", "temps",
            "min_sweeps")


def _fetched(res):
    return {k: (v.view(np.int32) if v.dtype == np.uint32 else v)
            for k, v in res.items()}


def run(state):
    c, seed = state["case"], state["seed"]
    kind = c["kind"]
    if kind == "solver":
        np.random.seed(seed % 2**32)  # the initial states' generator
        rows = state["solver"].metropolis_update(
            num_sweeps=c["sweeps"], num_reads=c["reads"],
            num_replicas=c["replicas"], min_temp=c["tmin"],
            max_temp=c["tmax"], update_strategy=c["update"],
            get_part_fun=c["partition"], seed=seed)
        cols = _COLUMNS + (("log_Zf",) if c["partition"] else ())
        return {k: np.stack([np.asarray(r[k]) for r in _rows(rows)])
                for k in cols}
    if kind in ("batch", "uneven", "lattice"):
        b = state["batch"]
        b.set_states(state["words"])
        b.run(c["sweeps"], seed=seed, update=c["update"])
        return _fetched(b.fetch())
    if kind == "rbm":
        m = state["rbm"]
        m.update_states_with_pysa(seed=seed)
        return {"v_state": m.v_state, "h_state": m.h_state}
    if kind == "ais_batch":
        out = run_ais_batch("ising", state["instances"], state["temps"],
                            seed=seed, update=c["update"])
        return {"samples": np.stack([s for s, _ in out]),
                "log_weights": np.stack([w for _, w in out])}
    if kind == "ais":
        np.random.seed(seed % 2**32)
        logz, samples, weights = state["solver"].annealed_importance(
            c["temps"], c["samples"], c["reference"],
            update_strategy=c["update"],
            reference_args=(0.4,) if c["reference"] == "bernoulli" else None,
            beta=c["beta"], seed=seed)
        return {"log_Zf": logz, "samples": samples,
                "weights": np.asarray(weights)}
    b, prop = state["batch"], state["prop"]
    b.set_states(state["words"])
    run_with_proposals(b, prop, c["sweeps"], seed=seed, interval=10,
                       train_every=5, train_pairs=10**9, min_accept=0.0)
    out = {k: prop.t[k] for k in ("w1", "b1", "w2", "b2", "loss")}
    out.update(logits=prop.t["z2"], spins=b.spins, energies=b.energies,
               best_energy=b.best_energy)
    return out


def _rows(frame):
    """The frame's rows as dicts, whether pandas is there or not."""
    return frame.to_dict("records") if hasattr(frame, "to_dict") else frame


# ---------------------------------------------------------------------- work
def work(case):
    """Bytes: couplings read once, states in, results out.  Operations: one
    random number and one decision per attempt (counted as 64: the ten
    Philox rounds shared by four attempts, the logarithm and the compare),
    plus the network's products for the learned proposal; the field updates
    of accepted flips depend on the data and are left out."""
    kind = case["kind"]
    if kind == "rbm":
        n = case["visible"] + case["hidden"]
        c = case["state_size"]
        return {"bytes": 4.0 * (case["visible"] * case["hidden"] + n) + 8.0 * c * n,
                "flops": 64.0 * c * n * case["steps"]}
    if kind in ("ais", "ais_batch"):
        I, n = case.get("instances", 1), case["n"]
        c = I * case["samples"]
        return {"bytes": 4.0 * I * n * n + 8.0 * c * n + 8.0 * c,
                "flops": 64.0 * c * n * case["temps"]}
    chains = case["replicas"] * case["reads"]
    if kind == "uneven":
        I = case["instances"]
        ns = [case["nmin"] + (case["nmax"] - case["nmin"]) * i // max(I - 1, 1)
              for i in range(I)]
        return {"bytes": sum(4.0 * n * n + chains * (3.0 * n / 8 + 16)
                             for n in ns),
                "flops": 64.0 * chains * sum(ns) * case["sweeps"]}
    n = case["side"] ** 2 if kind == "lattice" else case["n"]
    I = case["instances"] if kind == "learned" else 1
    couplings = 8.0 * 4 * n if kind == "lattice" else 4.0 * n * n
    # Solver takes and returns states as floats, PTBatch as bits
    per_spin = 5.0 if kind == "solver" else 3.0 / 8
    w = {"bytes": I * (couplings + chains * (per_spin * n + 16)),
         "flops": 64.0 * I * chains * n * case["sweeps"]}
    if kind == "learned":
        # per sweep: 0.2 training steps (three products each way of the two
        # layers) and 0.1 proposals (two forward passes, J delta)
        nn, hid, rd = n, case["hidden"], case["reads"]
        steps, props = case["sweeps"] // 5, case["sweeps"] // 10
        w["flops"] += 2.0 * I * rd * nn * (steps * 5 * hid +
                                           props * (4 * hid + nn))
        # weights and both Adam moments read and written by every step
        w["bytes"] += steps * 24.0 * I * 2 * nn * hid
    return w


# --------------------------------------------------------------------- exact
# Plain 64-bit restatement of the update rules on the same counter-based
# streams, one visited spin at a time over all chains.  Only for couplings
# whose fields are exact in float32 (integers, or integers times a power of
# two), so that the decisions are the same in both precisions.
_MASK = 0xFFFFFFFF
_TAG_SWEEP, _TAG_PT, _TAG_PERM, _TAG_AIS = 0, 1, 2, 3


def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 on int64 tensors holding 32-bit words."""
    k0, k1 = seed & _MASK, (seed >> 32) & _MASK
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & _MASK, (k1 + 0xBB67AE85) & _MASK
        p0, p1 = 0xD2511F53 * c0, 0xCD9E8D57 * c2
        c0, c1, c2, c3 = (((p1 >> 32) & _MASK) ^ c1 ^ k0, p1 & _MASK,
                          ((p0 >> 32) & _MASK) ^ c3 ^ k1, p0 & _MASK)
    return c0, c1, c2, c3


def _words(seed, tag, a, b, count, dev):
    """Draws 0 .. count - 1 of the streams (tag, instance 0, a, b[k]) as
    [len(b), count] 32-bit words."""
    q = torch.arange((count + 3) // 4, device=dev)[None, :]
    b = b[:, None].to(torch.int64)
    z = torch.zeros_like(q + b)
    w = _philox(z + q, z + a, z + b, z + tag, seed)
    return torch.stack(w, dim=2).reshape(b.shape[0], -1)[:, :count]


def _log_u(words):
    return torch.log((words.double() + 0.5) * 2.0**-32)


def _order(update, n, seed, sweep):
    if update != "random":
        return list(range(n))
    x = _words(seed, _TAG_PERM, sweep, torch.zeros(1, dtype=torch.int64), n,
               torch.device("cpu"))[0].tolist()
    p = list(range(n))
    for i in range(n - 1, 0, -1):
        j = (x[i] * (i + 1)) >> 32
        p[i], p[j] = p[j], p[i]
    return p


def _exact_pt(case, seed):
    ising = case["ptype"] == "ising"
    n, R, Rd = case["n"], case["replicas"], case["reads"]
    dev = torch.device("cuda")
    P = _matrix(case["values"], n, _gen(seed)).double()
    h = torch.diag(P).clone()
    J = P - torch.diag(h)
    rs = np.random.RandomState(seed % 2**32)
    x0 = np.stack([rs.randint(2, size=(R, n)) for _ in range(Rd)])
    s = torch.from_numpy(x0).to(dev).double().reshape(Rd * R, n)
    s = 2 * s - 1 if ising else s
    if case["partition"]:
        ratio = np.exp(1 / (R - 2) * np.log(case["tmax"] / case["tmin"]))
        betas = np.array([1 / (case["tmin"] * ratio**k) for k in range(R - 1)]
                         + [0.0], np.float32)
    elif R == 2:
        betas = np.array([1 / case["tmin"], 1 / case["tmax"]], np.float32)
    else:
        ratio = np.exp(1 / (R - 1) * np.log(case["tmax"] / case["tmin"]))
        betas = np.array([1 / (case["tmin"] * ratio**k) for k in range(R)],
                         np.float32)
    F = s @ J.T + h
    E = (s * (0.5 * (s @ J.T) + h)).sum(1)
    slot = np.tile(np.arange(R), (Rd, 1))       # slot -> replica
    best = E.clone()
    chains = torch.arange(Rd * R, device=dev)
    order_up = np.argsort(betas, kind="stable")
    log_omega = np.zeros((Rd, case["sweeps"]))
    for t in range(case["sweeps"]):
        beta = np.empty((Rd, R))
        np.put_along_axis(beta, slot, np.tile(betas.astype(np.float64),
                                              (Rd, 1)), 1)
        beta = torch.from_numpy(beta).to(dev).reshape(-1)
        lu = _log_u(_words(seed, _TAG_SWEEP, t, chains, n, dev))
        for k, i in enumerate(_order(case["update"], n, seed, t)):
            si = s[:, i]
            dn = 2 * si * F[:, i] if ising else (2 * si - 1) * F[:, i]
            acc = (dn >= 0) | (lu[:, k] < beta * dn)
            step = -2 * si if ising else 1 - 2 * si
            d = torch.where(acc, step, torch.zeros_like(step))
            E = E - torch.where(acc, dn, torch.zeros_like(dn))
            F += d[:, None] * J[i][None, :]
            s[:, i] += d
        best = torch.minimum(best, E)
        e = E.reshape(Rd, R).cpu().numpy().astype(np.float32)
        x = _words(seed, _TAG_PT, t, torch.arange(Rd), max(R - 1, 1),
                   torch.device("cpu")).numpy()
        for k in range(R - 1):
            k1, k2 = R - k - 1, R - k - 2
            r = np.arange(Rd)
            b1, b2 = slot[r, k1].copy(), slot[r, k2].copy()
            de = (e[r, b1] - e[r, b2]) * (betas[k1] - betas[k2])
            u = (x[:, k].astype(np.float64) + 0.5) * 2.0**-32
            sw = (de >= 0) | (u < np.exp(np.minimum(de, 0).astype(np.float64)))
            slot[r, k1] = np.where(sw, b2, b1)
            slot[r, k2] = np.where(sw, b1, b2)
        old = 0.0
        for q in order_up[1:]:
            b = float(betas[q])
            log_omega[:, t] -= (b - old) * e[np.arange(Rd), slot[:, q]]
            old = b
    with np.errstate(divide="ignore"):
        temps = 1 / betas.astype(np.float64)[slot]
    out = {k: None for k in _COLUMNS}
    out.update(energies=E.reshape(Rd, R).cpu().numpy(), temps=temps,
               best_energy=best.reshape(Rd, R).min(dim=1).values.cpu().numpy())
    if case["partition"]:
        m = log_omega.max(1)
        out["log_Zf"] = (m + np.log(np.exp(log_omega - m[:, None]).mean(1)) +
                         n * math.log(2))
    return out


def _exact_ais(case, seed):
    ising = case["ptype"] == "ising"
    n, ns = case["n"], case["samples"]
    dev = torch.device("cuda")
    J = case["beta"] * _matrix("pm1", n, _gen(seed)).double()
    rs = np.random.RandomState(seed % 2**32)
    p = 0.4
    bern = case["reference"] == "bernoulli"
    if bern:
        x0 = np.array([[rs.binomial(1, 1 - p) for _ in range(n)]
                       for _ in range(ns)])
    else:
        x0 = np.array([rs.randint(2, size=n) for _ in range(ns)])
    s = torch.from_numpy(x0).to(dev).double()
    s = 2 * s - 1 if ising else s
    F = s @ J
    E = 0.5 * (s * F).sum(1)
    lw = torch.zeros(ns, dtype=torch.float64, device=dev)
    lr = math.log((1 - p) / p) if bern else 0.0
    logp, log1p = math.log(p), math.log(1 - p)
    temps = np.array([(i + 1) / case["temps"] for i in range(case["temps"])],
                     np.float32)
    old = 0.0
    idx = torch.arange(ns, device=dev)
    for t, b in enumerate(temps.astype(np.float64)):
        lu = _log_u(_words(seed, _TAG_AIS, t, idx, n, dev))
        for k, i in enumerate(_order(case["update"], n, seed, t)):
            si = s[:, i]
            up = si > 0.5
            dn = 2 * si * F[:, i] if ising else (2 * si - 1) * F[:, i]
            ref = torch.where(up, torch.full_like(dn, -lr),
                              torch.full_like(dn, lr))
            full = b * dn + (1 - b) * ref
            acc = (full >= 0) | (lu[:, k] < full)
            step = -2 * si if ising else 1 - 2 * si
            d = torch.where(acc, step, torch.zeros_like(step))
            E = E - torch.where(acc, dn, torch.zeros_like(dn))
            F += d[:, None] * J[i][None, :]
            s[:, i] += d
        lw -= (b - old) * E
        if bern:
            ones = (s > 0.5).sum(1).double()
            lw -= (old - b) * -((n - ones) * logp + ones * log1p)
        old = b
    lw = lw.cpu().numpy()
    m = lw.max()
    w = np.exp(lw - m)
    return {"log_Zf": m + math.log(w.mean()) + (0 if bern else n * math.log(2)),
            "samples": None, "weights": w / w.sum()}


def exact(case, seed):
    # one visited spin costs about 0.2 ms here; real couplings round
    # differently in 64 bits and their chains part ways
    if case["kind"] == "solver" and case["values"] != "normal" and \
            case["n"] * case["sweeps"] <= 20000:
        return _exact_pt(case, seed)
    if case["kind"] == "ais" and case["n"] * case["temps"] <= 20000:
        return _exact_ais(case, seed)
    return None
