"""Dynamic E4M3 quantisation at its edges: values on and beside the midpoints of the E4M3 grid, the subnormal range, scales
near the ends of the float range, ragged counts."""
from __future__ import annotations

import pytest
import torch

from aginfer_b200.recipes import Tensor, U32
from aginfer_b200.recipes.layout import padded_token_rows, unpack_kblock_swizzled
from oracle import ops
from tests.gpu_util import run_recipe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def values(count: int, kind: str) -> torch.Tensor:
    g = torch.Generator().manual_seed(count)
    if kind == "bits":           # every exponent down to 2^-60 of the largest
        x = torch.randn(count, generator=g) * torch.exp2(torch.randint(-60, 1, (count,), generator=g).float())
    elif kind == "grid":         # multiples of fractions of the E4M3 grid's steps: many of them midpoints
        x = torch.randint(-28672, 28673, (count,), generator=g).float() / 64 * torch.exp2(torch.randint(-12, 1, (count,), generator=g).float())
        x[0] = 448.0
    else:                        # scales near the ends of the float range
        x = torch.randn(count, generator=g) * (1e-36 if kind == "tiny" else 1e36)
    return x.to(BF)


@pytest.mark.parametrize("kind", ["bits", "grid", "tiny", "huge"])
@pytest.mark.parametrize("count", [7, 16, 4104, 262152, 5 * 262144 + 24])
def test_quantize_matches_the_division(tmp_path, count, kind):
    x = values(count, kind)
    want, scale = ops.quantize_e4m3(x)

    def body(r):
        s = r.alloc(4)
        r.quantize_e4m3(Tensor("x"), Tensor("q"), s, count)
        r.launch("agi_copy_u32", (1, 1, 1), (32, 1, 1), [s, Tensor("scale"), U32(1)])

    got, _ = run_recipe(tmp_path, {}, {"x": x}, {"q": (torch.float8_e4m3fn, (count,)), "scale": (torch.int32, (1,))}, body)
    assert got["scale"].item() == scale.reshape(1).view(torch.int32).item()
    assert torch.equal(got["q"].view(torch.uint8), want.view(torch.uint8))


@pytest.mark.parametrize("rows,cols", [(1, 128), (9, 384), (129, 2048), (300, 1408)])
def test_packed_quantize_matches_the_row_major_one(tmp_path, rows, cols):
    x = values(rows * cols, "grid").reshape(rows, cols)
    want, _ = ops.quantize_e4m3(x)
    blocks = cols // 128, padded_token_rows(rows)

    def body(r):
        q, s = r.alloc(blocks[0] * blocks[1] * 128), r.alloc(4)
        r.quantize_e4m3(Tensor("x"), q, s, rows * cols, packed=(rows, cols))
        r.launch("agi_copy_u32", (64, 1, 1), (256, 1, 1), [q, Tensor("q"), U32(blocks[0] * blocks[1] * 32)])

    got, _ = run_recipe(tmp_path, {}, {"x": x}, {"q": (torch.float8_e4m3fn, (*blocks, 128))}, body)
    assert torch.equal(unpack_kblock_swizzled(got["q"].view(torch.uint8), rows), want.view(torch.uint8))
