"""Sums over an instance's rows with the preconditioners whose instances never share a cluster:
one pass over the rows, as many as there are (a row or two per thread, many, a remainder), against
the oracle's exact solution.  A Krylov cycle takes many Arnoldi steps here, so a sum that missed or
repeated rows would not converge."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [dict(precond="segment"), dict(precond="jacobi", max_iter=4000),
                                  dict(krylov="bicgstab", precond="tree")],
                         ids=["segment", "jacobi", "bicgstab-tree"])
def test_batch_of_sizes(gpu, pkg, orc, model, opts):
    specs = [model.random_tree(seed=31 + q, n_target=n, dt=2.5e-5, tspan=1e-3)
             for q, n in enumerate((60, 255, 300, 1025, 2100))]
    b = pkg.Batch([pkg.ProblemArrays.from_spec(sp, pkg.derive(sp)) for sp in specs], mode=1,
                  precision="fp64", tol=1e-11, tol_mode="rel", restart=30,
                  **{"max_iter": 2000, **opts})
    b.set_runs([(1, 9, sp.init_time, sp.end_input) for sp in specs])
    b.advance(8)
    V, st = b.snapshot_all(), b.instance_stats()
    b.close()
    assert (st["nonconverged"] == 0).all()
    for v, sp in zip(V, specs):
        Vo, _, _, _ = orc.implicit_run(sp, orc.derive(sp), sp.dt_abs, 1, 9, linsolve=0)
        assert np.abs(v - Vo).max() < 1e-9
