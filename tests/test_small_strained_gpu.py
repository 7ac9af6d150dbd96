"""A small strained mixed pack (below 8192 elements) takes one launch per step in calls of up to 128
steps and several per launch in longer ones: alternating between the two, with probes and a strain
ramp, gives every bit of one launch per step throughout."""
import pytest

from test_block_gpu import compare, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("calls", [(64, 200, 64, 133, 64), (200, 3, 128, 129, 65)])
def test_alternating_calls(gpu, pkg, model, calls):
    specs = [model.random_tree(seed=70, n_target=1501), model.myelinated_axon(n_nodes=3)]
    assert sum(sp.n for sp in specs) < 8192
    compare(pkg, specs, problems(pkg, specs), calls, True, "mixed")
