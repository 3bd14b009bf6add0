"""Rotary embedding a row per block (`agi_mrope_pair_bf16`), the kernel that aligned arena operands take: one or two
tensors, 1-D and three-stream positions, frequency ladders, more vectors than the block's threads hold at once, and
columns beside the heads that must stay as they are."""
from __future__ import annotations

import pytest
import torch

from aginfer_b200.recipes import Tensor, U32
from oracle import ops
from tests.gpu_util import run_recipe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
# one bf16 step in the top binade where a rounding falls the other way (2^-7 of the largest value), and the angle: at
# positions up to 600, three fp32 roundings of 2^-24 each on frequency and product
TOL = 2.0 ** -7 + 600 * 3 * 2.0 ** -24


def randn(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(BF)


def turned(tmp_path, parts, positions, emit):
    """``parts``: name -> (tensor, heads, head_dim); every tensor is copied into the arena, turned there by ``emit`` and
    copied out.  Returns the outputs and asserts that the row kernel, and no other rotary kernel, ran."""
    kernels = []

    def body(r):
        at = {}
        for name, (x, _, _) in parts.items():
            words = x.numel() // 2
            at[name] = r.alloc(x.numel() * 2)
            r.launch("agi_copy_u32", (64, 1, 1), (256, 1, 1), [Tensor(name), at[name], U32(words)])
        before = r.launch_count()
        emit(r, at)
        kernels.extend(launch["kernel"] for launch in r.profiles[0].launches[before:])
        for name, (x, _, _) in parts.items():
            r.launch("agi_copy_u32", (64, 1, 1), (256, 1, 1), [at[name], Tensor(f"{name}_out"), U32(x.numel() // 2)])

    inputs = {name: x for name, (x, _, _) in parts.items()}
    if positions is not None:
        inputs["pos"] = positions
    got, _ = run_recipe(tmp_path, {}, inputs, {f"{n}_out": (BF, x.shape) for n, (x, _, _) in parts.items()}, body)
    assert kernels == ["agi_mrope_pair_bf16"]
    return got


def check(got, parts, want_of):
    for name, (x, heads, d) in parts.items():
        rows, out = x.shape[0], got[f"{name}_out"]
        want = want_of(x[:, :heads * d].reshape(rows, heads, d)).reshape(rows, -1)
        assert torch.equal(out[:, heads * d:], x[:, heads * d:])
        assert ops.max_rel_err(out[:, :heads * d], want) <= TOL, name


@pytest.mark.parametrize("rows,heads,spare,d,offset", [(1, 1, 0, 16, 0), (5, 3, 8, 48, 7), (50, 32, 0, 48, 256), (3, 2, 16, 256, 500),
                                                       (288, 18, 256, 128, 0)])
def test_one_tensor_one_stream(tmp_path, rows, heads, spare, d, offset):
    parts = {"x": (randn(rows, heads * d + spare, seed=rows + d), heads, d)}
    got = turned(tmp_path, parts, None, lambda r, at: r.rope(at["x"], rows, heads, d, heads * d + spare, 1e6, pos_offset=offset))
    check(got, parts, lambda x: ops.rope(x, 1e6, offset))


@pytest.mark.parametrize("rows,hq,hk,d", [(50, 8, 4, 128), (7, 28, 4, 128), (2, 40, 3, 128), (1, 1, 1, 32)])
def test_two_tensors_one_stream(tmp_path, rows, hq, hk, d):
    parts = {"q": (randn(rows, hq * d + 64, seed=1), hq, d), "k": (randn(rows, hk * d, seed=2), hk, d)}
    got = turned(tmp_path, parts, None, lambda r, at: r.rope_pair(at["q"], hq, hq * d + 64, at["k"], hk, hk * d, rows, d, 1e4, pos_offset=88))
    check(got, parts, lambda x: ops.rope(x, 1e4, 88))


@pytest.mark.parametrize("rows,hq,hk,d,sections,ladder", [
    (101, 16, 2, 128, (16, 24, 24), None), (64, 28, 4, 128, (16, 24, 24), None), (65, 32, 0, 80, (20, 20, 0), 20),
    (3, 2, 2, 64, (0, 0, 32), None), (9, 33, 5, 128, (64, 0, 0), None), (6, 1, 1, 256, (50, 40, 38), 64)])
def test_three_position_streams(tmp_path, rows, hq, hk, d, sections, ladder):
    positions = torch.randint(0, 600, (3, rows), generator=torch.Generator().manual_seed(8), dtype=torch.int32)
    parts = {"q": (randn(rows, hq * d + 32, seed=3), hq, d)}
    if hk:
        parts["k"] = (randn(rows, hk * d, seed=4), hk, d)
    got = turned(tmp_path, parts, positions, lambda r, at: r.mrope(
        at["q"], Tensor("pos"), rows, hq, d, hq * d + 32, 1e6, sections, ladder=ladder,
        second=(at["k"], hk, hk * d) if hk else None))
    check(got, parts, lambda x: ops.mrope(x, positions, 1e6, sections, ladder))
