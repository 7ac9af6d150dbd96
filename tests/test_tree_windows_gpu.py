"""The implicit kernel's windowed tree sweeps (csrc/tree.cuh, csrc/refine.cuh) at the sizes
where they can go wrong: trees that end one row before, on and after a window edge, row counts
that are no multiple of the rows per thread, cables cut into many pieces, one-row pieces next
to branch points, and trees with more pieces than a CTA's shared memory holds.

FP64 is held to 1e-9 V against the oracle's exact solution (the bar of the implicit tests).
The mixed-precision step (fused passes, Richardson cycles) is held to 1e-8 V against the same
solver with GMRES refinement cycles, which go through separate passes: both stop at a residual
of 1e-10 of the right-hand side."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WIN = 1024
FP64 = dict(tol=1e-11, tol_mode="rel", restart=30)
MIXED = dict(precision="mixed", restart=20, tol=1e-10, tol_mode="rel")


def cable(model, n):  # n elements in all: the root, n - 2 compartments, the end
    return model.straight_axon(n_comp=n - 2, length=2e-6 * (n - 2), dt=2.5e-5, tspan=1e-3)


def tree(model, name):
    if name.startswith("cable"):
        return cable(model, int(name[5:]))
    if name == "twigs":  # 4095 branches of 2 to 4 compartments: more pieces than fit
        return model.random_binary_tree(depth=11, seed=4, len_lo=2e-6, len_hi=4e-6, dt=2.5e-5,
                                        tspan=1e-3)
    seed, n = name.split("x")
    return model.random_tree(seed=int(seed), n_target=int(n), dt=2.5e-5, tspan=1e-3)


TREES = ["cable5", "cable128", "cable129", "cable%d" % (WIN - 1), "cable%d" % WIN, "cable%d" % (WIN + 1),
         "cable%d" % (WIN + 2), "cable%d" % (5 * WIN + 3), "3x701", "8x2050", "11x6001", "twigs"]


def run(pkg, cls, spec, steps, **opts):
    s = cls(pkg.ProblemArrays.from_spec(spec, pkg.derive(spec)), **opts)
    s.run(1, 1 + steps, spec.init_time, spec.end_input)
    V, st = s.snapshot(), s.stats()
    s.close()
    assert st.nonconverged_steps == 0
    return V


@pytest.mark.parametrize("scheme", ["be", "cn"])
@pytest.mark.parametrize("name", TREES)
def test_one_tree(gpu, pkg, orc, model, name, scheme):
    spec = tree(model, name)
    steps = 12
    V = run(pkg, pkg.SolverIm, spec, steps, scheme=scheme, **FP64)
    Vo, _, _, _ = orc.implicit_run(spec, orc.derive(spec), spec.dt_abs, 1, 1 + steps, linsolve=0,
                                   scheme=int(scheme == "cn"))
    assert np.abs(V - Vo).max() < 1e-9
    a = run(pkg, pkg.SolverIm, spec, steps, scheme=scheme, **MIXED)
    b = run(pkg, pkg.SolverIm, spec, steps, scheme=scheme, refinement="gmres", **MIXED)
    assert np.abs(a - b).max() < 1e-8


# trees around a warp's window (128 rows) and the rows' chunks of 128, and trees whose pieces do
# and do not all fit the staging of a block's walk
SMALL = ["cable%d" % n for n in (4, 127, 128, 129, 130, 255, 257, 1151)] + \
    ["5x%d" % n for n in (60, 130, 900, 1500, 2100, 2700, 3400)]


@pytest.mark.parametrize("names,copies", [(["cable5", "twigs", "71x4117"] + TREES, 1), (SMALL, 1),
                                          (SMALL, 24)], ids=["all", "small", "small360"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_of_all(gpu, pkg, orc, model, precision, names, copies):
    """The same trees in one batch (instances start on multiples of four rows), with trees of
    more pieces than shared memory holds at several places in it.  Batches of few trees give each
    a cluster, of many (copies) a CTA."""
    specs = [tree(model, n) for n in names] * copies
    probs = [pkg.ProblemArrays.from_spec(sp, pkg.derive(sp)) for sp in specs]
    steps = 12
    out = {}
    for refinement in ("auto", "gmres") if precision == "mixed" else ("auto",):
        b = pkg.Batch(probs, mode=1, refinement=refinement,
                      **(FP64 if precision == "fp64" else MIXED))
        b.set_runs([(1, 1 + steps, sp.init_time, sp.end_input) for sp in specs])
        b.advance(steps)
        out[refinement] = b.snapshot_all()
        for q in range(len(specs)):
            np.testing.assert_array_equal(out[refinement][q], b.snapshot(q))
        assert (b.instance_stats()["nonconverged"] == 0).all()
        b.close()
    for q, sp in enumerate(specs):
        if q >= len(names):
            np.testing.assert_array_equal(out["auto"][q], out["auto"][q - len(names)])
        elif precision == "mixed":
            assert np.abs(out["auto"][q] - out["gmres"][q]).max() < 1e-8
        else:
            Vo, _, _, _ = orc.implicit_run(sp, orc.derive(sp), sp.dt_abs, 1, 1 + steps, linsolve=0)
            assert np.abs(out["auto"][q] - Vo).max() < 1e-9


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [40, WIN, 1500])
def test_trees_next_to_one_that_overflowed(gpu, pkg, model, precision, n):
    """Rows of different trees lie next to each other: a tree whose potential is not finite leaves
    its neighbours' results as they are, bit for bit."""
    sp = cable(model, n)
    d = pkg.derive(sp)
    opts = dict(mode=1, precision=precision, tol=1e-10, tol_mode="rel")
    got = []
    for bad in (False, True):
        ends = pkg.ProblemArrays.from_spec(sp, d, V0=np.full(n, np.inf)) if bad else \
            pkg.ProblemArrays.from_spec(sp, d)
        b = pkg.Batch([ends, pkg.ProblemArrays.from_spec(sp, d), ends], **opts)
        b.set_runs([(1, 13, sp.init_time, sp.end_input)] * 3)
        b.advance(12)
        got.append(b.snapshot(1))
        b.close()
    assert np.isfinite(got[0]).all()
    np.testing.assert_array_equal(got[0], got[1])
