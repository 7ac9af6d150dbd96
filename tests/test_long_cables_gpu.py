"""FP64 implicit batches of cables that a warp's windows (128 rows) cut into more pieces than the
staged walk holds: a block's (307 pieces) and a cluster's (all its numbers in device memory beyond
819), against the oracle's exact solution; and snapshots of trees of very different sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule", [1, 0], ids=["block", "cluster"])
def test_long_cables(gpu, pkg, orc, model, schedule):
    specs = [model.straight_axon(n_comp=n - 2, length=2e-6 * (n - 2), dt=2.5e-5, tspan=1e-3)
             for n in (45001, 110002, 39297, 130)]
    b = pkg.Batch([pkg.ProblemArrays.from_spec(sp, pkg.derive(sp)) for sp in specs], mode=1,
                  precision="fp64", tol=1e-11, tol_mode="rel", restart=30, schedule=schedule)
    b.set_runs([(1, 7, sp.init_time, sp.end_input) for sp in specs])
    b.advance(6)
    V = b.snapshot_all()
    assert (b.instance_stats()["nonconverged"] == 0).all()
    for q, sp in enumerate(specs):
        np.testing.assert_array_equal(V[q], b.snapshot(q))
        Vo, _, _, _ = orc.implicit_run(sp, orc.derive(sp), sp.dt_abs, 1, 7, linsolve=0)
        assert np.abs(V[q] - Vo).max() < 1e-9
    b.close()
