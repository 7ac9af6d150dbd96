"""Several explicit steps per launch (csrc/block.cu), mixed precision and FP64: every result
equals the per-step kernels' (tiled = 0) bit for bit -- potentials, gates, the other potential
buffer, samples and spikes -- over the sizes and calls where the tiles can go wrong: packs of
one tile and of many, trees whose branches are shorter than a halo, mostly passive trees, runs
that end inside a launch, calls that are no multiple of a launch or of a captured chunk, probes
on sealed ends and on neighbouring elements, and a strain ramp over tile edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def trees(model, name):
    if name.startswith("axon") and len(name) > 4:
        n = int(name[4:])
        return [model.straight_axon(n_comp=n, length=1e-5 * n, dtf=0.8)]
    if name == "axon":
        return [model.straight_axon(n_comp=9000, length=9e-2, dtf=0.8)]
    if name == "myelin":
        return [model.myelinated_axon(n_nodes=12)]
    if name == "twigs":  # branches of 2 to 4 compartments
        return [model.random_binary_tree(depth=11, seed=4, len_lo=2e-6, len_hi=4e-6)]
    if name == "few":
        return [model.random_tree(seed=90 + q, n_target=n) for q, n in enumerate((700, 401, 350))]
    if name == "tree":
        return [model.random_tree(seed=5, n_target=30011)]
    return [model.random_tree(seed=70 + q, n_target=n) for q, n in
            enumerate((1501, 9000, 2999, 640, 12007))] + [model.myelinated_axon(n_nodes=3)]


def problems(pkg, specs):
    out = []
    for k, sp in enumerate(specs):
        d = pkg.derive(sp)
        V = sp.rest_pot + 0.03 * np.sin(np.arange(sp.n) * 0.011 + k) ** 2  # activity everywhere
        t = sp.terminals[1:]
        V[t] = V[sp.mother[t]]
        V[0] = V[1]
        out.append(pkg.ProblemArrays.from_spec(sp, d, 0.8 * d.dT_crit, V0=V))
    return out


def run(pkg, specs, probs, calls, strain, precision, **opts):
    b = pkg.Batch(probs, precision=precision, **opts)
    if strain:
        sp = specs[-1]
        b.set_strain(len(specs) - 1, sp, np.arange(sp.n // 3, sp.n // 3 + 900), 0.0, 0.2, 0.0,
                     300 * probs[-1].dT)
    pr = []
    for q, sp in enumerate(specs):
        mid = sp.n // 2
        pr += [(q, 1), (q, mid), (q, mid + 1), (q, mid), (q, int(sp.terminals[-1])), (q, 0)]
    b.record(pr, interval=4, capacity=64, threshold=-0.05, max_spikes=8)
    total = sum(calls)
    ends = [1 + total - 13 * q for q in range(len(specs))]
    b.set_runs([(1, e, 0.0, 40 * p.dT) for e, p in zip(ends, probs)])
    for n in calls:
        b.advance(n)
    states = [b.get_state(q) for q in range(len(specs))]
    rec = b.recording()
    snap = b.snapshot_all()
    b.close()
    return states, rec, snap


@pytest.mark.parametrize("name,strain", [("axon", False), ("myelin", False), ("myelin", True),
                                         ("twigs", False), ("tree", False), ("batch", False),
                                         ("batch", True)])
@pytest.mark.parametrize("calls", [(3, 200), (64, 65, 130), (257,), (64, 200, 64, 133, 64, 64)])
def test_blocks_equal_single_steps(gpu, pkg, model, name, strain, calls):
    specs = trees(model, name)
    probs = problems(pkg, specs)
    compare(pkg, specs, probs, calls, strain, "mixed")


# one and two rounds of eight-lane elements, one-thread elements, several tiles per SM
@pytest.mark.parametrize("name", ["axon300", "axon1000", "few", "axon3000", "axon9000", "twigs",
                                  "tree", "batch"])
@pytest.mark.parametrize("calls", [(3, 70), (64, 65)])
def test_fp64_blocks_equal_single_steps(gpu, pkg, model, name, calls):
    specs = trees(model, name)
    compare(pkg, specs, problems(pkg, specs), calls, False, "fp64")


def compare(pkg, specs, probs, calls, strain, precision):
    (a, ra, va) = run(pkg, specs, probs, calls, strain, precision)
    (b, rb, vb) = run(pkg, specs, probs, calls, strain, precision, tiled=False)
    for x, y in zip(a, b):
        for part in ("V", "V_other", "m", "h", "n"):
            np.testing.assert_array_equal(getattr(x, part), getattr(y, part), err_msg=part)
    for x, y in zip(va, vb):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(ra.num_samples, rb.num_samples)
    np.testing.assert_array_equal(ra.num_spikes, rb.num_spikes)
    for x, y in zip(ra.values + ra.spikes, rb.values + rb.spikes):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("name", ["axon", "tree", "batch"])
def test_plan_built_later(gpu, pkg, model, name, precision):
    """Without recording the plan is built when calls have asked for 128 steps: runs that begin
    with one launch per step and go on with several end as those that keep to one."""
    specs = trees(model, name)
    probs = problems(pkg, specs)
    out = []
    for opts in ({}, {"tiled": False}):
        b = pkg.Batch(probs, precision=precision, **opts)
        b.set_runs([(1, 1000, 0.0, 40 * p.dT) for p in probs])
        for n in (40, 64, 20, 64, 3, 200, 64):
            b.advance(n)
        out.append([b.get_state(q) for q in range(len(specs))])
        b.close()
    for x, y in zip(*out):
        for part in ("V", "V_other", "m", "h", "n"):
            np.testing.assert_array_equal(getattr(x, part), getattr(y, part), err_msg=part)
