"""Mixed-precision implicit batches whose trees take different ways through a step: some end
with the Richardson cycles, some stall there and go on with GMRES, whose basis lies in the
workspace that all trees share.  No tree's result depends on what its neighbours do, or on when.

A cable of 3 nm compartments stalls: its rows' terms cancel by eight digits (conductance to
capacitance 1.4e8), so FP64 rounding holds its residual near 1e-8 of the right-hand side, a
hundred times the tolerance.  The other trees' (1e-14 and less) end below it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPTS = dict(mode=1, precision="mixed", restart=8, tol=1e-10, tol_mode="rel", max_iter=12)
STEPS = 6


def specs_of(model):
    stiff = [model.straight_axon(n_comp=n - 2, length=3e-9 * (n - 2), dt=2.5e-5, tspan=1e-3)
             for n in (1030, 1500, 4099)]
    easy = [model.random_tree(seed=60 + q, n_target=n, dt=2.5e-5, tspan=1e-3)
            for q, n in enumerate((1100, 2051, 9000))]
    return [easy[0], stiff[0], easy[2], stiff[1], easy[1], stiff[2]]


def run(pkg, specs, **opts):
    b = pkg.Batch([pkg.ProblemArrays.from_spec(sp, pkg.derive(sp)) for sp in specs], **OPTS, **opts)
    b.set_runs([(1, 1 + STEPS, sp.init_time, sp.end_input) for sp in specs])
    b.advance(STEPS)
    V, pc = b.snapshot_all(), b.pass_counts()
    b.close()
    return V, pc


@pytest.mark.parametrize("shape,copies", [({"schedule": 1}, 1), ({"schedule": 1}, 60), ({}, 1), ({}, 60)],
                         ids=["block", "block-many", "cluster", "many"])
def test_trees_that_reach_gmres_next_to_trees_that_do_not(gpu, pkg, model, shape, copies):
    specs = specs_of(model)
    alone = [run(pkg, [sp], schedule=1) for sp in specs]
    gmres = np.array([pc["basis"][0] > 0 for _, pc in alone])
    np.testing.assert_array_equal(gmres, [q % 2 == 1 for q in range(len(specs))])
    V, pc = run(pkg, specs * copies, **shape)
    again, _ = run(pkg, specs * copies, **shape)
    for q in range(len(V)):
        k = q % len(specs)
        np.testing.assert_array_equal(V[q], again[q])   # whatever ran beside it
        np.testing.assert_array_equal(V[q], V[k])       # wherever it lies
        assert np.isfinite(V[q]).all()
        if shape:  # one CTA per tree, as alone
            np.testing.assert_array_equal(V[q], alone[k][0][0])
            assert pc["basis"][q] == alone[k][1]["basis"][0]


def test_a_tree_does_not_depend_on_its_company(gpu, pkg, model):
    """The number of trees and the largest of them decide whether a tree has one CTA or a cluster of
    2, 4 or 8, and how many CTAs an SM holds: the potential and the residual's norm that ends a step
    are the same bits in all of them (windows and chunks of windows depend on the tree alone)."""
    base = [model.random_tree(seed=80 + q, n_target=n, dt=2.5e-5, tspan=1e-3)
            for q, n in enumerate((900, 1500, 2600, 9000, 30000))]
    probs = [pkg.ProblemArrays.from_spec(sp, pkg.derive(sp)) for sp in base]
    opts = dict(mode=1, precision="mixed", restart=20, tol=1e-10, tol_mode="rel")

    def go(which, **shape):
        b = pkg.Batch([probs[q] for q in which], **opts, **shape)
        b.set_runs([(1, 1 + STEPS, base[q].init_time, base[q].end_input) for q in which])
        b.advance(STEPS)
        V, st = b.snapshot_all(), b.instance_stats()
        b.close()
        assert (st["nonconverged"] == 0).all()
        return V, st["last_residual"]

    ref, res = go(range(5), schedule=1)  # a CTA each
    small = [0, 1, 2]
    for which, shape in (([0, 1], {}), ([0, 2, 1], {}), (list(range(5)), {}), (list(range(5)) * 10, {}),
                         (small * 30, {}), (small * 60, {}), (small * 170, {}),
                         (list(range(5)), {"tile_ctas_per_sm": 4}), (small * 30, {"tile_ctas_per_sm": 2}),
                         (list(range(5)) * 10, {"schedule": 1})):
        V, r = go(which, **shape)
        for k, q in enumerate(which):
            np.testing.assert_array_equal(V[k], ref[q], err_msg=f"{len(which)} trees {shape}")
            assert r[k] == res[q], (len(which), shape, k)
