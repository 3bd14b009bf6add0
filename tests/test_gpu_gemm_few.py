"""The tensor-core GEMM for few tokens: K over the ranks of a cluster, or its slices left to the norm that reads them."""
import pytest
import torch

from aginfer_b200.recipes import Tensor, Weight
from aginfer_b200.recipes.builder import TS_MAX_SLICES, ts_tiling
from oracle import ops
from tests.gpu_util import run_recipe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
# One rounding to bf16 of values up to the largest output: half a step of its binade, 2^-9 of it, and as much again for
# the rounding of an intermediate (gate, residual sum); fp32 sums in another order stay three digits below.
TOL = 2 ** -8


def randn(*shape, seed, std=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * std).to(BF)


# tokens at the edges of 8-row groups and 16-column units; features that fill no tile; one K block, ragged K slices
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 33, 50, 63, 64])
@pytest.mark.parametrize("N,K,act,extras", [(1536, 1536, None, "bias res"), (6144, 1536, "gelu_tanh", "bias"), (200, 704, "silu", ""),
                                            (67, 64, "relu", "bias res"), (1536, 6144, None, "")])
def test_products_of_few_tokens(tmp_path, M, N, K, act, extras):
    x, w = randn(M, K, seed=1), randn(N, K, seed=2, std=K ** -0.5)
    weights, inputs = {"w": w}, {"x": x}
    if "bias" in extras:
        weights["b"] = randn(N, seed=3, std=0.1)
    if "res" in extras:
        inputs["res"] = randn(M, N, seed=4)

    def body(r):
        r.gemm_few(Tensor("x"), [(Weight("w"), Weight("b") if "b" in weights else None, Tensor("y"), N, N)], M, K, act=act,
                   residual=Tensor("res") if "res" in inputs else None)
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, weights, inputs, {"y": (BF, (M, N)), "status": (torch.int32, (1,))}, body, repeats=2)
    want = ops.gemm(x, w, bias=weights.get("b"), residual=inputs.get("res"), act=act)
    assert got["status"].item() == 0 and ops.max_rel_err(got["y"], want) < TOL


@pytest.mark.parametrize("M", [1, 9, 50, 64])
@pytest.mark.parametrize("I,K", [(4096, 1024), (96, 128)])
def test_swiglu_of_few_tokens(tmp_path, M, I, K):
    x, gate, up = randn(M, K, seed=1), randn(I, K, seed=2, std=K ** -0.5), randn(I, K, seed=3, std=K ** -0.5)

    def body(r):
        r.gemm_swiglu(Tensor("x"), (Weight("g"), None, None), (Weight("u"), None, None), Tensor("y"), M, I, K)
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, {"g": gate, "u": up}, {"x": x}, {"y": (BF, (M, I)), "status": (torch.int32, (1,))}, body, repeats=2)
    g, u = ops.gemm(x, gate), ops.gemm(x, up)
    want = (torch.nn.functional.silu(g.float()) * u.float()).to(BF)
    assert got["status"].item() == 0 and ops.max_rel_err(got["y"], want) < 2 * TOL      # gate and up are rounded too


@pytest.mark.parametrize("M,cols,K", [(1, 128, 64), (17, 1536, 1536), (17, 1536, 6144), (50, 1024, 4096), (64, 2048, 704)])
@pytest.mark.parametrize("norm", ["layer", "adaln", "rms"])
def test_a_norm_adds_the_slices_of_a_split_product(tmp_path, M, cols, K, norm):
    x, w, bias, res = randn(M, K, seed=1), randn(cols, K, seed=2, std=K ** -0.5), randn(cols, seed=3, std=0.1), randn(M, cols, seed=4)
    mod = randn(2 * cols, seed=5, std=0.3)
    assert ts_tiling(M, (cols,), K, 2, split=True)["slices"] <= TS_MAX_SLICES

    def body(r):
        partial = r.alloc(TS_MAX_SLICES * M * cols * 4)
        slices = r.gemm_split(Tensor("x"), [(Weight("w"), cols)], partial, M, K)
        if norm == "rms":
            r.rmsnorm_sum(Tensor("res"), partial, Weight("b"), Weight("mod"), Tensor("out"), Tensor("y"), M, cols, slices)
        else:
            r.layernorm_sum(Tensor("res"), partial, Weight("b"), Tensor("out"), Tensor("y"), M, cols, slices,
                            **({"scale": Weight("mod"), "shift": Weight("mod") + 2 * cols} if norm == "adaln" else {}))
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, {"w": w, "b": bias, "mod": mod}, {"x": x, "res": res},
                        {"out": (BF, (M, cols)), "y": (BF, (M, cols)), "status": (torch.int32, (1,))}, body, repeats=2)
    assert got["status"].item() == 0
    assert ops.max_rel_err(got["out"], ops.gemm(x, w, bias=bias, residual=res)) < TOL
    out = got["out"]          # what the norm saw
    want = (ops.rmsnorm(out, mod[:cols]) if norm == "rms" else
            ops.layernorm(out, 1e-5, mod[:cols], mod[cols:]) if norm == "adaln" else ops.layernorm(out, 1e-5))
    assert ops.max_rel_err(got["y"], want) < TOL
