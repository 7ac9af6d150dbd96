"""Performance cases of the solver hot path, through the public Python interface.

A case is a simulation in progress: one tree (`SolverEx` / `SolverIm`) or a batch of trees
(`Batch`) whose potential and gates are somewhere between rest and a spike, with the
stimulus on.  One pass advances it by a number of loop iterations and reads the potential
back, as a program that monitors a run does; a pass on the same state continues the run.

Sizes: the 1 cm squid axon, the myelinated axon with its strain ramp, the depth-10 binary
tree (Crank-Nicolson) and the random-tree population (1e3 to 1e5 compartments, log-uniform)
of the benchmark, and trees of the sizes that the tests and the server use in between.
"""
from __future__ import annotations

import ctypes
import dataclasses
import functools
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("168861_gb300")
model = pkg.model
check = pkg.solver.check

EXPLICIT, IMPLICIT = 0, 1  # nrt_mode
SHAPES = 96                # distinct trees of a population (larger ones repeat them)
DT_IMPLICIT = 2.5e-5


def _case(name, mode, shape, precision, steps, n=0, count=1, loop=False, probes=0, strain=False,
          scheme="be", tol=1e-10, tree_seed=1):
    c = dict(mode=mode, shape=shape, precision=precision, steps=steps, n=n, count=count, loop=loop,
             probes=probes, strain=strain, scheme=scheme, tol=tol, tree_seed=tree_seed)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the reference's own use: one short unmyelinated axon in double precision, spikes
        # recorded at three places along it
        _case("axon-explicit-fp64", "explicit", "axon", "fp64", 512, n=1000, probes=3),
        # the drop-in loop of the reference's driver: update() and calculate() called from
        # the host for every step of a small dendritic tree
        _case("tree1500-loop-explicit-fp64", "explicit", "random", "fp64", 64, n=1500, loop=True,
              tree_seed=11),
        # a large dendritic tree in double precision (a ragged size; a run that does not end
        # on a whole number of graph replays)
        _case("tree65k-explicit-fp64", "explicit", "random", "fp64", 200, n=65000, tree_seed=12),
        # the strained myelinated axon: 200 nodes of Ranvier, mostly passive compartments
        _case("myelin-strain-explicit-mixed", "explicit", "myelin", "mixed", 640, n=200,
              strain=True, probes=4),
        # what the server packs together: a few trees at a time
        _case("batch24-explicit-mixed", "explicit", "population", "mixed", 256, n=10000, count=24,
              tree_seed=13),
        # the population, explicit: larger than L2 many times over
        _case("batch1024-explicit-mixed", "explicit", "population", "mixed", 64, n=100000,
              count=1024, tree_seed=14),
        # the drop-in loop of the implicit solver with its default (the reference's) tolerance
        _case("axon-loop-implicit-fp64", "implicit", "axon", "fp64", 24, n=1000, loop=True, tol=0.0),
        # the depth-10 binary tree (2047 branches, about 257,000 compartments), Crank-Nicolson
        _case("binary10-implicit-cn-fp64", "implicit", "binary", "fp64", 8, n=10, scheme="cn"),
        # one mid-size tree in mixed precision on the whole GPU (a request of its own in the server)
        _case("tree30k-implicit-mixed", "implicit", "random", "mixed", 32, n=30000, tree_seed=15),
        # a micro-batch in double precision
        _case("batch48-implicit-fp64", "implicit", "population", "fp64", 8, n=10000, count=48,
              tree_seed=16),
        # the population, implicit mixed precision: the benchmark's headline workload
        _case("batch2048-implicit-mixed", "implicit", "population", "mixed", 8, n=100000,
              count=2048, tree_seed=17),
    ]


# how much one compartment-step weighs in draw()'s bound on a case's cost
_WEIGHT = {("explicit", "mixed"): 1, ("explicit", "fp64"): 8, ("implicit", "mixed"): 8,
           ("implicit", "fp64"): 30}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    mode = rng.choice(["explicit", "explicit", "implicit", "implicit"])
    precision = rng.choice(["fp64", "mixed"])
    shape = rng.choice(["axon", "random", "random", "population", "population", "binary"] +
                       (["myelin"] if mode == "explicit" else ["random"]))
    count, n = 1, 0
    if shape == "axon":
        n = _log_int(rng, 300, 20000)
        elems = n
    elif shape == "random":
        n = _log_int(rng, 800, 200000)
        elems = n
    elif shape == "binary":
        n = rng.randint(3, 10)
        elems = 125 << (n + 1)
    elif shape == "myelin":
        n = _log_int(rng, 4, 200)
        elems = 1000 * n
    else:
        count, n = _log_int(rng, 2, 400), _log_int(rng, 3000, 100000)
        elems = count * n // 4
    loop = shape in ("axon", "random") and elems < 3000 and rng.random() < 0.4
    steps = rng.randint(16, 48) if loop else (_log_int(rng, 48, 700) if mode == "explicit"
                                              else _log_int(rng, 4, 48))
    budget = 1.2e9
    steps = max(4, min(steps, int(budget / (elems * _WEIGHT[mode, precision]))))
    return _case(None, mode, shape, precision, steps, n=n, count=count, loop=loop,
                 probes=rng.choice([0, 0, 1, 5]) if count == 1 and not loop else 0,
                 strain=shape == "myelin" and rng.random() < 0.6,
                 scheme=rng.choice(["be", "be", "cn"]) if mode == "implicit" else "be",
                 tree_seed=rng.randint(1, 10 ** 6))


# ---------------------------------------------------------------- inputs

def _hops(spec):
    """Compartments between each element and the root."""
    j = np.arange(spec.n)
    brk = np.concatenate([[0], np.nonzero(spec.mother[1:] != j[:-1])[0] + 1])
    hops = np.zeros(spec.n, np.int64)
    for a, b in zip(brk, list(brk[1:]) + [spec.n]):
        h = 0 if spec.mother[a] < 0 else hops[spec.mother[a]] + 1
        hops[a:b] = h + np.arange(b - a)
    return hops


@functools.lru_cache(maxsize=1)
def _specs(shape, n, count, seed):
    """The trees of a case with their derived parameters and distances from the root."""
    if shape == "axon":
        specs = [model.straight_axon(n_comp=n, length=1e-5 * n, dtf=0.8)]
    elif shape == "myelin":
        specs = [model.myelinated_axon(n_nodes=n)]
    elif shape == "binary":
        specs = [model.random_binary_tree(depth=n, seed=seed)]
    elif shape == "random":
        specs = [model.random_tree(seed=seed, n_target=n)]
    else:
        k = min(count, SHAPES)
        lo = 1000.0
        u = (np.arange(k) + 0.5) / k  # every part of the range, the largest tree among them
        sizes = np.exp(math.log(lo) + u * (math.log(max(n, 2 * lo)) - math.log(lo))).astype(int)
        order = np.random.default_rng(seed).permutation(k)
        specs = [model.random_tree(seed=seed + int(i), n_target=int(sizes[i])) for i in order]
    return [(s, pkg.derive(s), _hops(s)) for s in specs]


def _trees(c):
    return _specs(c["shape"], c["n"], c["count"] if c["shape"] == "population" else 1,
                  c["tree_seed"])


def _rates(lib, v, p):
    """The six HH rates at potential v (V), parameters p (ls_Na, ls_K, rest)."""
    vna, vk = ((v + p[0]) - p[2]) / 1e-3, ((v + p[1]) - p[2]) / 1e-3
    return ((2.5 - 0.1 * vna) / (lib.exp(2.5 - 0.1 * vna) - 1), 4 * lib.exp(-vna / 18),
            0.07 * lib.exp(-vna / 20), 1 / (lib.exp(3 - 0.1 * vna) + 1),
            (0.1 - 0.01 * vk) / (lib.exp(1 - 0.1 * vk) - 1), 0.125 * lib.exp(-vk / 80))


def _strain_segment(c, spec):
    """The strained compartments: a fortieth of the axon in its middle."""
    if not c["strain"]:
        return np.zeros(0, np.int32)
    mid, half = spec.n // 2, max(1, spec.n // 80)
    return np.arange(mid - half, mid + half, dtype=np.int32)


def _problems(c, seed):
    """The problems of a case: a wave of depolarisation along every distinct tree, gates at
    their steady state for it, and a stimulus current for every problem, drawn from the seed."""
    rng = np.random.default_rng(seed)
    trees = _trees(c)
    waves, out = [], []
    for spec, d, hops in trees:
        amp, length, phase = rng.uniform(0.01, 0.045), rng.uniform(150, 600), rng.uniform(0, math.pi)
        V = spec.rest_pot + amp * np.sin(hops * (math.pi / length) + phase) ** 2
        t = spec.terminals[1:]
        V[t] = V[spec.mother[t]]  # sealed ends copy their neighbours
        V[0] = V[1]
        hp = d.hparam.copy()
        if d.num_hh:
            a = _rates(np, V[d.hh_elem], (hp[9], hp[10], hp[11]))
            for q in range(3):
                hp[q] = a[2 * q] / (a[2 * q] + a[2 * q + 1])
        waves.append((V, hp))
    for k in range(c["count"]):
        (spec, d, _), (V, hp) = trees[k % len(trees)], waves[k % len(trees)]
        dT = 0.8 * d.dT_crit if c["mode"] == "explicit" else \
            (1e-5 if c["scheme"] == "cn" else DT_IMPLICIT)
        inp = np.zeros(spec.n)
        inp[1] = rng.uniform(0.5e-9, 3e-9)
        spec = dataclasses.replace(spec, input_current=inp)
        out.append((spec, pkg.ProblemArrays.from_spec(spec, d, dT, V0=V, hparam=hp)))
    return out


def _options(c):
    o = dict(precision=c["precision"])
    if c["mode"] == "implicit":
        o.update(scheme=c["scheme"])
        if c["tol"] > 0:
            o.update(tol=c["tol"], tol_mode="rel", restart=30 if c["precision"] == "fp64" else 20,
                     max_iter=2000)
    return o


def prepare(case, seed):
    made = _problems(case, seed)
    probs = [p for _, p in made]
    sizes = [p.num_elem for p in probs]
    out = torch.empty(sum(sizes), dtype=torch.float64, pin_memory=True)
    state = dict(case=case, i=1, out=out, V=out.numpy())
    if case["count"] == 1:
        s = (pkg.SolverEx if case["mode"] == "explicit" else pkg.SolverIm)(probs[0], **_options(case))
        spec = made[0][0]
        seg = _strain_segment(case, spec)
        if len(seg):  # 0 -> 20 % over 5 ms
            s.set_strain(spec, seg, 0.0, 0.2, 0.0, 5e-3)
        if case["probes"]:
            el = np.linspace(1, spec.n - 2, case["probes"]).astype(np.int32)
            s.record(el, interval=15, capacity=512, threshold=-0.05)
    else:
        s = pkg.Batch(probs, mode=EXPLICIT if case["mode"] == "explicit" else IMPLICIT,
                      **_options(case))
        s.set_runs([(1, 1 << 40, 0.0, 10.0)] * case["count"])
    state["solver"] = s
    return state


def run(state):
    c, s = state["case"], state["solver"]
    if c["count"] > 1:
        s.advance(c["steps"])
        check(s.lib.nrt_batch_snapshot_all(
            s.h, state["V"].ctypes.data_as(ctypes.POINTER(ctypes.c_double))), "snapshot_all")
        return {"V": state["out"]}
    if c["loop"]:
        for _ in range(c["steps"]):
            s.update(True)
            s.calculate()
    else:
        s.run(state["i"], state["i"] + c["steps"], 0.0, 10.0)
        state["i"] += c["steps"]
    s.snapshot(state["V"])
    res = {"V": state["out"]}
    if c["probes"]:
        r = s.recording()
        res.update(samples=r.num_samples, spikes=r.num_spikes,
                   values=np.concatenate(r.values))
    return res


def work(case):
    trees = _trees(case)
    n = nh = 0
    for k in range(case["count"]):
        spec, d, _ = trees[k % len(trees)]
        n += spec.n
        nh += d.num_hh
    b = 8 if case["precision"] == "fp64" else 4
    # state in and out (potential, gates), coefficients and the tree in, potential out
    bytes_ = n * (16 + 2 * b + 4 + 8) + nh * 6 * b
    # per compartment-step: the stencil or the assembly and the tree solve; per channel
    # compartment six exponentials, three quotients, three gates and two currents
    per = (14 if case["mode"] == "explicit" else 40, 130)
    return {"bytes": bytes_, "flops": case["steps"] * (per[0] * n + per[1] * nh)}


# ---------------------------------------------------------------- 64-bit results

class _Pack:
    """All trees of a case as one set of FP64 arrays on the GPU."""

    def __init__(self, c, seed):
        made = _problems(c, seed)
        off = np.cumsum([0] + [p.num_elem for _, p in made])
        dev = "cuda"
        cat = lambda f, dt: torch.from_numpy(np.concatenate(  # noqa: E731
            [np.asarray(f(s, p, o), dt) for (s, p), o in zip(made, off)])).to(dev)
        a = lambda k, dt=np.float64: cat(lambda s, p, o: p.arrays[k], dt)  # noqa: E731
        ix = lambda k: cat(lambda s, p, o: p.arrays[k] + o, np.int64)  # noqa: E731
        self.n = int(off[-1])
        self.mother = cat(lambda s, p, o: np.maximum(p.arrays["mother"], 0) + o, np.int64)
        self.dr, self.dl, self.br = ix("dr"), ix("dl"), a("branching")
        term = ix("terminals")
        root = torch.from_numpy(off[:-1].astype(np.int64)).to(dev)
        self.term = torch.zeros(self.n, dtype=torch.bool, device=dev)
        self.term[term] = True
        self.root, self.last = root, torch.from_numpy(off[1:].astype(np.int64) - 1).to(dev)
        self.src = self.mother.clone()
        self.src[root] = root + 1
        self.dx, self.cm, self.ra = a("dx"), a("c_m"), a("r_a")
        self.W, self.K, self.inp, self.V = a("W"), a("K"), a("input"), a("V0")
        self.dT = cat(lambda s, p, o: np.full(p.num_elem, p.dT), np.float64)
        self.hh = ix("hh_elem")
        self.g = {k: a(k) for k in ("m", "h", "n", "g_Na", "g_K", "G_L", "E_Na", "E_K", "E_L",
                                    "ls_Na", "ls_K", "rest")}
        self.hops = cat(lambda s, p, o: _hops(s), np.int64)
        self.gax = 1.0 / (self.ra * self.dx)

    def gates(self):
        if not len(self.hh):
            return
        g, dt = self.g, self.dT[self.hh] * 1000
        r = _rates(torch, self.V[self.hh], (g["ls_Na"], g["ls_K"], g["rest"]))
        for q, k in enumerate("mhn"):
            g[k] = g[k] + dt * (r[2 * q] * (1 - g[k]) - r[2 * q + 1] * g[k])
        na, k_ = g["g_Na"] * g["m"] ** 3 * g["h"], g["g_K"] * g["n"] ** 4
        self.W[self.hh] = -(na + k_ + g["G_L"])
        self.K[self.hh] = na * g["E_Na"] + k_ * g["E_K"] + g["G_L"] * g["E_L"]

    def explicit(self):
        self.gates()
        V = self.V
        f = (V[self.dr] - V) * self.gax[self.dr] + (V[self.mother] - V) * self.gax
        f = f + self.br * (V[self.dl] - V) * self.gax[self.dl]
        f = f + self.W * self.dx * V + self.K * self.dx + self.inp
        V = V + self.dT / (self.cm * self.dx) * f
        self.V = torch.where(self.term, V[self.src], V)

    def implicit(self, old, cn, order):
        """One step by elimination from the leaves to the root and back (order: the rows of
        each distance from the root); `old` is the potential one step back, which the rows
        that carry no equation take."""
        self.gates()
        V = self.V
        ident = self.term.clone()
        ident[self.root] = True
        ident[self.last] = True
        j = torch.arange(self.n, device=V.device)
        first = torch.zeros_like(ident)
        first[self.root + 1] = True
        gm = torch.where(first | ident, 0.0, self.gax)  # to the mother
        s = 2.0 if cn else 1.0
        cmt = self.cm * self.dx / self.dT
        c = s * cmt - self.W * self.dx
        nxt = torch.clamp(j + 1, max=self.n - 1)
        gr = torch.where(ident | ident[nxt], 0.0, self.gax[nxt])
        gl = torch.where(ident, 0.0, self.br * self.gax[self.dl])
        d = c + gm + gr + gl
        if cn:
            b = (2 * cmt + self.W * self.dx) * V - gm * (V - V[self.mother]) - gr * (V - V[nxt])
            b = b - gl * (V - V[self.dl]) + 2 * (self.K * self.dx + self.inp)
        else:
            b = cmt * V + self.K * self.dx + self.inp
        for rows in reversed(order):
            m, w = self.mother[rows], gm[rows] / d[rows]
            d.index_add_(0, m, -w * gm[rows])
            b.index_add_(0, m, w * b[rows])
        x = torch.zeros_like(V)
        for rows in order:
            x[rows] = (b[rows] + gm[rows] * x[self.mother[rows]]) / d[rows]
        self.V = torch.where(ident, old, x)


def exact(case, seed):
    if case["strain"]:
        return None  # the strained coefficients come from the parameter pipeline
    trees = _trees(case)
    n = sum(trees[k % len(trees)][0].n for k in range(case["count"]))
    depth = max(int(h.max()) for _, _, h in trees)
    if case["mode"] == "explicit":
        if case["steps"] * (2e-3 + 5e-10 * 20 * n) > 12:
            return None
    elif case["steps"] * depth * 1.6e-4 > 12 or n > 4e6:
        return None
    p = _Pack(case, seed)
    el = np.linspace(1, n - 2, case["probes"]).astype(np.int64) if case["probes"] else []
    at = [int(p.src[e]) if bool(p.term[e]) and case["mode"] == "explicit" else int(e) for e in el]
    vals = []
    order = None
    if case["mode"] == "implicit":
        ident = p.term.cpu().numpy().copy()
        ident[p.root.cpu().numpy()] = True
        ident[p.last.cpu().numpy()] = True
        rows = np.nonzero(~ident)[0]
        h = p.hops.cpu().numpy()[rows]
        rows = rows[np.argsort(h, kind="stable")]
        cut = np.cumsum(np.bincount(h, minlength=depth + 1))[:-1]
        order = [torch.from_numpy(r).cuda() for r in np.split(rows, cut) if len(r)]
    old = p.V
    for i in range(1, 1 + case["steps"]):
        now = p.V
        if order is None:
            p.explicit()
        else:
            p.implicit(old, case["scheme"] == "cn", order)
        old = now
        if i % 16 == 0:
            vals.append([float(p.V[e]) for e in at])
    res = {"V": p.V}
    if case["probes"]:
        res.update(samples=None, spikes=None,
                   values=np.asarray(vals, np.float64).reshape(-1, len(at)).T.reshape(-1).copy())
    return res
