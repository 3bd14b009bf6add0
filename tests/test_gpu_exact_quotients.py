"""Quotients by a corrected reciprocal are the division's, bit for bit: SwiGLU over every bf16 gate, E4M3 quantisation of every
bf16 value for amax from one end of the range to the other."""
import pytest
import torch

from aginfer_b200.recipes import Tensor, U32
from oracle import ops
from tests.gpu_util import run_recipe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
EVERY = torch.arange(65536, dtype=torch.int32).to(torch.uint16).view(BF)


def test_swiglu_of_every_gate_equals_the_silu_that_divides(tmp_path):
    def body(r):
        r.swiglu(Tensor("gate"), Tensor("one"), Tensor("y"), 64, 1024, 1024)
        r.launch("agi_silu_bf16", (256, 1, 1), (256, 1, 1), [Tensor("gate"), Tensor("want"), U32(65536)])

    got, _ = run_recipe(tmp_path, {}, {"gate": EVERY, "one": torch.ones(65536, dtype=BF)},
                        {"y": (BF, (65536,)), "want": (BF, (65536,))}, body)
    same = got["y"].view(torch.int16) == got["want"].view(torch.int16)
    assert (same | (got["y"].isnan() & got["want"].isnan())).all()


@pytest.mark.parametrize("exponent", [-126, -100, -79, -78, -20, 0, 7, 60, 87, 90, 127])
@pytest.mark.parametrize("mantissa", [1.0, 1.3359375, 1.9921875])
def test_quantisation_of_every_value_up_to_amax(tmp_path, exponent, mantissa):
    amax = torch.tensor(mantissa * 2.0 ** exponent, dtype=BF)
    x = torch.where(EVERY.abs() <= amax, EVERY, amax)       # NaN: amax

    def body(r):
        r.quantize_e4m3(Tensor("x"), Tensor("q"), r.alloc(4), 65536)

    got, _ = run_recipe(tmp_path, {}, {"x": x}, {"q": (torch.float8_e4m3fn, (65536,))}, body)
    want, _ = ops.quantize_e4m3(x)
    assert torch.equal(got["q"].view(torch.uint8), want.view(torch.uint8))
