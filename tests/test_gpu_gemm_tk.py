"""The tensor-core GEMM with tokens as the MMA's A operand, at the edges of its tiles: token groups of 8 ... 512 rows, one
to ten K runs, clusters, ragged N, every epilogue, packed and row-major operands."""
from __future__ import annotations

import pytest
import torch

from aginfer_b200.recipes import Tensor, Weight
from aginfer_b200.recipes.layout import pack_kblock_swizzled, padded_token_rows
from oracle import ops
from tests.gpu_util import run_recipe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16

CASES = [
    (33, 256, 512, "bf16", "plain"), (65, 272, 1024, "bf16", "bias_res"), (127, 2048, 5504, "e4m3", "res"),
    (128, 96, 128, "e4m3", "bias"), (129, 1000, 2048, "bf16", "bias_gelu"), (77, 2048, 2048, "e4m3", "bias"),
    (101, 1024, 11008, "e4m3", "plain"), (257, 1536, 640, "packed", "bias_res"), (513, 144, 3456, "packed", "bias"),
    (300, 130, 256, "packed", "bias_gelu"), (1100, 384, 256, "e4m3", "plain"),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_gemm_tk_edges(tmp_path, case):
    check_against_the_oracle(tmp_path, case)


@pytest.mark.parametrize("kind", ["bf16", "e4m3", "packed"])
def test_gemm_tk_of_more_than_8192_rows(tmp_path, kind):
    check_against_the_oracle(tmp_path, (8201, 144, 256, kind, "bias_res"))


def check_against_the_oracle(tmp_path, case):
    M, N, K, kind, epi = case
    g = torch.Generator().manual_seed(M + N + K)
    x, wf = torch.randn(M, K, generator=g).to(BF), torch.randn(N, K, generator=g) * 0.02
    bias = (torch.randn(N, generator=g) * 0.1).to(BF) if "bias" in epi else None
    res = torch.randn(M, N, generator=g).to(BF) if "res" in epi else None
    act = "gelu_tanh" if "gelu" in epi else None
    kw = dict(bias=bias, residual=res, act=act)
    weights, inputs = {}, {"x": x}
    if kind == "bf16":
        weights["w"], want = wf.to(BF), ops.gemm(x, wf.to(BF), **kw)
    else:
        (wq, ws), (xq, xs) = ops.quantize_e4m3(wf.to(BF)), ops.quantize_e4m3(x)
        weights.update({"w": pack_kblock_swizzled(wq) if kind == "packed" else wq, "s": ws.reshape(())})
        want = ops.gemm(xq, wq, scale_a=xs, scale_w=ws, **kw)
    if bias is not None:
        weights["b"] = bias
    if res is not None:
        inputs["res"] = res

    def body(r):
        kw = dict(bias=Weight("b") if bias is not None else None, residual=Tensor("res") if res is not None else None,
                  act=act, tactic="tcgen05_plan")
        if kind == "bf16":
            r.gemm(Tensor("x"), Weight("w"), Tensor("y"), M, N, K, **kw)
        else:
            packed = kind == "packed"
            q, s = r.alloc((padded_token_rows(M) if packed else M) * K), r.alloc(4)
            r.quantize_e4m3(Tensor("x"), q, s, M * K, packed=(M, K) if packed else None)
            r.gemm(q, Weight("w"), Tensor("y"), M, N, K, dtype="e4m3", scale_a=s, scale_w=Weight("s"), packed=packed, **kw)
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, weights, inputs, {"y": (BF, (M, N)), "status": (torch.int32, (1,))}, body, repeats=2)
    assert got["status"].item() == 0, hex(got["status"].item())
    assert ops.max_rel_err(got["y"], want) < 1e-2
