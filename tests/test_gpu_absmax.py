"""max |x| in one launch against torch: lengths around a vector of eight, a block's vectors and the loop's stride."""
import pytest
import torch

from aginfer_b200.recipes import Tensor, U32
from tests.gpu_util import run_recipe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("count,blocks", [(1, 1), (9, 1), (255 * 8 + 7, 1), (256 * 8, 1), (4 * 256 * 8, 1), (7 * 256 * 8 + 1, 1),
                                          (8 * 256 * 8 - 3, 1), (5 * 592 * 256 * 8 + 1001, 592)])
@pytest.mark.parametrize("at", [0.0, 0.5, 1.0])
def test_absmax_finds_the_largest_wherever_it_is(tmp_path, count, blocks, at):
    x = torch.randn(count, generator=torch.Generator().manual_seed(count)).to(BF)
    x[torch.arange(0, count, 5)] = float("nan")         # a NaN never is the maximum
    x[int(at * (count - 1))] = -300.0

    def body(r):
        r.launch("agi_absmax_bf16", (blocks, 1, 1), (256, 1, 1), [Tensor("x"), U32(count), Tensor("amax")])

    got, _ = run_recipe(tmp_path, {}, {"x": x}, {"amax": (torch.float32, (1,))}, body)
    assert got["amax"].item() == 300.0
