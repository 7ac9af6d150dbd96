"""What the autotuner times is what a tuned batch runs: its shapes keep the several-step launches and
the clusters on, and explicit shapes are timed over calls long enough to use them."""
import importlib
import time

import pytest

at = importlib.import_module("168861_gb300.autotune")
lib = importlib.import_module("168861_gb300._lib")


class Tree:
    num_elem = 5000


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_explicit_shapes_are_timed_over_long_calls(monkeypatch, precision):
    """Small mixed packs take several steps per launch in calls of more than 128 steps."""
    seen = []

    def timer(ps, mode, prec, ov, steps, warmup, runs=None, **opts):
        seen.append(steps)
        return 1.0

    monkeypatch.setattr(at, "time_candidate", timer)
    at.tune([Tree()] * 4, lib.NRT_EXPLICIT, precision, cache="", device_key="dev")
    assert seen and min(seen) > 128


def test_time_candidate_runs_an_untimed_call_first(monkeypatch):
    """A first call makes the several-step plan: it is not timed."""
    solver = importlib.import_module("168861_gb300.solver")
    calls = []

    class Fake:
        def __init__(self, *a, **k):
            pass

        def set_runs(self, runs):
            self.end = min(e for _, e, _, _ in runs)

        def advance(self, n):
            calls.append(n)
            time.sleep(0.05 if sum(calls) <= 300 else 0.001)  # the plan is made within 300 steps

        def synchronize(self):
            pass

        def close(self):
            assert sum(calls) <= self.end - 1  # the runs are long enough

    monkeypatch.setattr(solver, "Batch", Fake)
    per = at.time_candidate([Tree()], lib.NRT_EXPLICIT, "mixed", {}, steps=300, warmup=0)
    assert len(calls) >= 3 and per < 0.01 / 300


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1000, 9000])
def test_step_threads_keep_several_steps_per_launch(gpu, pkg, model, n):
    sp = model.straight_axon(n_comp=n, length=1e-5 * n, dtf=0.8)
    d = pkg.derive(sp)
    p = pkg.ProblemArrays.from_spec(sp, d, 0.8 * d.dT_crit)
    count = {}
    for ov in [{}] + at.candidates(lib.NRT_EXPLICIT, "fp64"):
        b = pkg.Batch([p], precision="fp64", **ov)
        b.set_runs([(1, 10000, 0.0, 1.0)])
        b.advance(512)
        b.synchronize()
        l0 = pkg.kernel_launches()
        b.advance(512)
        b.synchronize()
        count[str(ov)] = pkg.kernel_launches() - l0
        b.close()
    assert len(set(count.values())) == 1 and count["{}"] < 256, count
