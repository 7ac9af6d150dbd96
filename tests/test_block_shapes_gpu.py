"""Implicit batches of one CTA per tree: two, three or four CTAs on an SM (a rule by the trees'
sizes and number, or tile_ctas_per_sm) give the same trees bit for bit, and so do the halves of a
CTA that take a small tree's row chunks in turn."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP64 = dict(precision="fp64", tol=1e-11, tol_mode="rel", restart=30)
MIXED = dict(precision="mixed", tol=1e-10, tol_mode="rel", restart=20)


def run(pkg, specs, steps=8, **opts):
    b = pkg.Batch([pkg.ProblemArrays.from_spec(sp, pkg.derive(sp)) for sp in specs], mode=1, **opts)
    b.set_runs([(1, 1 + steps, sp.init_time, sp.end_input) for sp in specs])
    b.advance(steps)
    V, st = b.snapshot_all(), b.instance_stats()
    b.close()
    assert (st["nonconverged"] == 0).all()
    return V, st["last_residual"]


# trees that are too small for a CTA's warps, more than the usual CTAs take; trees of one size in
# fewer rounds; more trees than four CTAs per SM
@pytest.mark.parametrize("sizes,count", [((40, 130, 257, 510), 480), ((700, 701), 330), ((1025,), 610)])
@pytest.mark.parametrize("opts", [FP64, MIXED, dict(FP64, precond="segment", tol=1e-8, max_iter=2000)],
                         ids=["fp64", "mixed", "segment"])
def test_ctas_per_sm(gpu, pkg, orc, model, sizes, count, opts):
    base = [model.random_tree(seed=17 + q, n_target=n, dt=2.5e-5, tspan=1e-3)
            for q, n in enumerate(sizes)]
    specs = [base[q % len(base)] for q in range(count)]
    ref, rr = run(pkg, specs, **opts)
    for k in (1, 4):
        V, r = run(pkg, specs, tile_ctas_per_sm=k, **opts)
        for x, y in zip(ref, V):
            np.testing.assert_array_equal(x, y)
        np.testing.assert_array_equal(rr, r)
    for q, sp in enumerate(base):
        Vo, _, _, _ = orc.implicit_run(sp, orc.derive(sp), sp.dt_abs, 1, 9, linsolve=0)
        assert np.abs(ref[q] - Vo).max() < (1e-9 if opts is FP64 else 1e-6)
