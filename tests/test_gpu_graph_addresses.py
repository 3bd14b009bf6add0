"""Which passes replay a graph: the first set of addresses at once, further sets from their second pass on."""
from __future__ import annotations

import pytest
import torch

from aginfer_b200.recipes import RecipeBuilder, Tensor, io
from aginfer_b200.recipes.package import build_aim, describe
from aginfer_b200.runner import Runner

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sets,passes,graphs,replays", [(1, 3, 1, 3), (3, 1, 1, 1), (3, 3, 3, 7), (12, 1, 1, 1)])
def test_address_sets_get_a_graph_when_they_come_back(tmp_path, sets, passes, graphs, replays):
    weights = {"unused.pad": torch.zeros(8, dtype=torch.bfloat16)}
    recipe = RecipeBuilder(describe(weights))
    recipe.begin_profile("default", [io("left", "F32", [16]), io("right", "F32", [16])], [io("output", "F32", [16])])
    recipe.vector_add(Tensor("left"), Tensor("right"), Tensor("output"), 16)
    runner = Runner(build_aim(tmp_path, weights, recipe))
    tensors = [({"left": torch.full((16,), float(i), device="cuda"), "right": torch.ones(16, device="cuda")},
                {"output": torch.zeros(16, device="cuda")}) for i in range(sets)]
    for _ in range(passes):
        for inputs, outputs in tensors:
            outputs["output"].zero_()
            runner.run(inputs, outputs)
    torch.cuda.synchronize()
    for i, (_, outputs) in enumerate(tensors):
        assert torch.equal(outputs["output"].cpu(), torch.full((16,), i + 1.0))
    stats = runner.stats()
    assert stats["enqueues"] == sets * passes and stats["graphs_built"] == graphs and stats["graph_launches"] == replays
