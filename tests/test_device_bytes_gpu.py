"""nrt_stats.device_bytes counts all device memory of a handle -- the several-step plan with its
second gate buffer, recordings and strains as well as the arena -- and the server's estimate of a
request covers it.  The plan is there only where a call uses it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def batch(pkg, specs, **opts):
    probs = []
    for sp in specs:
        d = pkg.derive(sp)
        probs.append(pkg.ProblemArrays.from_spec(sp, d, 0.8 * d.dT_crit))
    b = pkg.Batch(probs, **opts)
    b.set_runs([(1, 10000, 0.0, 1.0)] * len(specs))
    return b


@pytest.mark.parametrize("precision,per", [("mixed", 12), ("fp64", 24)])
def test_plan_is_counted(gpu, pkg, model, precision, per):
    specs = [model.random_tree(seed=11, n_target=10000)]
    b = batch(pkg, specs, precision=precision)
    start = b.stats().device_bytes
    b.advance(2)
    assert b.stats().device_bytes == start      # too short for a plan
    b.advance(300)
    assert b.stats().device_bytes >= start + per * specs[0].n  # the second gate buffer and more
    b.close()


def test_no_plan_where_no_call_uses_it(gpu, pkg, model):
    sp = model.myelinated_axon(n_nodes=12)
    seg = np.arange(sp.n // 3, sp.n // 3 + 900)
    b = batch(pkg, [sp], precision="fp64")      # FP64 strain: one launch per step
    b.set_strain(0, sp, seg, 0.0, 0.2, 0.0, 1e-3)
    start = b.stats().device_bytes
    b.advance(300)
    assert b.stats().device_bytes == start
    b.close()
    b = batch(pkg, [sp], precision="mixed")     # ten recorded steps do not pay for one
    b.record([(0, 5), (0, sp.n // 2)], interval=1, capacity=64)
    start = b.stats().device_bytes
    b.advance(10)
    assert b.stats().device_bytes == start
    b.advance(400)
    assert b.stats().device_bytes > start
    b.close()


def test_recording_and_strain_are_counted(gpu, pkg, model):
    sp = model.myelinated_axon(n_nodes=12)
    b = batch(pkg, [sp], precision="mixed")
    start = b.stats().device_bytes
    b.record([(0, 5)], interval=1, capacity=5000)
    rec = b.stats().device_bytes
    assert rec >= start + 8 * 5000
    b.set_strain(0, sp, np.arange(500, 1500), 0.0, 0.2, 0.0, 1e-3)
    assert b.stats().device_bytes >= rec + 16 * 1000
    b.close()


@pytest.mark.parametrize("kind", ["random", "twigs", "cable"])
@pytest.mark.parametrize("implicit", [False, True])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_server_estimate_covers_a_request(gpu, pkg, model, kind, implicit, precision):
    dt = dict(dt=2.5e-5) if implicit else {}
    sp = model.random_tree(seed=9, n_target=60000, **dt) if kind == "random" else \
        model.straight_axon(n_comp=40000, length=2e-6 * 40000, **dt) if kind == "cable" else \
        model.random_binary_tree(depth=13, seed=4, len_lo=2e-6, len_hi=4e-6, **dt)
    d = pkg.derive(sp)
    p = pkg.ProblemArrays.from_spec(sp, d) if implicit else pkg.ProblemArrays.from_spec(sp, d, 0.8 * d.dT_crit)
    opts = dict(precision=precision)
    if implicit:
        opts.update(restart=20, tol=1e-8, tol_mode="rel")
    srv = pkg.Server(budget_bytes=4 << 30, implicit_opts=opts if implicit else dict(precision="mixed"),
                     explicit_opts=dict(precision="mixed") if implicit else opts)
    steps = 4 if implicit else 600
    rid = srv.submit(p, implicit, 1, 1 + steps, sp.init_time, sp.end_input)
    srv.drain()
    estimate = srv.stats().peak_bytes
    srv.result(rid)
    srv.close()
    b = pkg.Batch([p], mode=int(implicit), **opts)
    b.set_runs([(1, 1 + steps, sp.init_time, sp.end_input)])
    b.advance(steps)
    used = b.stats().device_bytes
    b.close()
    assert estimate >= used, (estimate, used)
