"""The order in which a tensor-core GEMM's tiles and token groups run changes where operands come from and nothing else: every
launch family, several groups and tiles, ragged edges, both orders bit for bit the same and right."""
import pytest
import torch

from aginfer_b200.recipes import Tensor, Weight, builder
from aginfer_b200.recipes.layout import pack_kblock_swizzled, padded_token_rows
from oracle import ops
from tests.gpu_util import run_recipe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("M,N,K", [(600, 300, 256), (1100, 1000, 640), (2100, 40, 128)])
def test_both_orders_give_the_same_product(tmp_path, monkeypatch, M, N, K):
    g = torch.Generator().manual_seed(M)
    x, w, w2 = [torch.randn(*s, generator=g) for s in ((M, K), (N, K), (N, K))]
    bias = torch.zeros(N, dtype=BF)
    (xq, xs), (wq, ws) = ops.quantize_e4m3(x.to(BF)), ops.quantize_e4m3((w * 0.02).to(BF))
    weights = {"a": w.to(BF), "b": w2.to(BF), "bias": bias, "q": wq, "p": pack_kblock_swizzled(wq), "ws": ws.reshape(())}
    bf, f8 = ("plain", "pair0", "pair1", "batch0", "batch1"), ("e4m3", "plan", "persistent")
    got, grids = {}, {}

    def body(r):
        y = {n: Tensor(n) for n in (*bf, "swiglu", *f8)}
        q, qp, s, two = r.alloc(M * K), r.alloc(padded_token_rows(M) * K), r.alloc(4), r.alloc(2 * M * N * 2)
        r.gemm(Tensor("x"), Weight("a"), y["plain"], M, N, K, tactic="tcgen05_plan")
        r.gemm_group(Tensor("x"), [(Weight("a"), None, None, y["pair0"], N, N), (Weight("b"), None, None, y["pair1"], N, N)], M, K)
        r.gemm_swiglu(Tensor("x"), (Weight("a"), None, None), (Weight("b"), None, None), y["swiglu"], M, N, K)
        r.gemm_batch(Tensor("x"), [(Weight("a"), Weight("bias")), (Weight("b"), Weight("bias"))], two, M, N, K, seg_stride=M * N)
        for i in range(2):
            r.launch("agi_copy_u32", (64, 1, 1), (256, 1, 1), [two + i * M * N * 2, y[f"batch{i}"], builder.U32(M * N // 2)])
        r.quantize_e4m3(Tensor("x"), q, s, M * K)
        r.quantize_e4m3(Tensor("x"), qp, s, M * K, packed=(M, K))
        fp8 = dict(dtype="e4m3", scale_a=s, scale_w=Weight("ws"))
        r.gemm(q, Weight("q"), y["e4m3"], M, N, K, tactic="tcgen05_plan", **fp8)
        r.gemm(qp, Weight("p"), y["plan"], M, N, K, tactic="tcgen05_plan", packed=True, **fp8)
        r.gemm(qp, Weight("p"), y["persistent"], M, N, K, tactic="persistent", packed=True, **fp8)
        r.export_status(Tensor("status"))
        grids[first] = [tuple(l["grid"]) for l in r.profiles[0].launches if l["kernel"].startswith("agi_gemm_tk_bf16")]

    for first in (True, False):
        monkeypatch.setattr(builder, "groups_first", lambda *a, **kw: first)
        out = {n: (BF, (M, N)) for n in (*bf, "swiglu", *f8)} | {"status": (torch.int32, (1,))}
        (tmp_path / str(first)).mkdir()
        got[first], _ = run_recipe(tmp_path / str(first), weights, {"x": x.to(BF)}, out, body)
        assert got[first]["status"].item() == 0
    assert [(b, a, c) for a, b, c in grids[True]] == grids[False]
    for n in (*bf, "swiglu", *f8):
        assert torch.equal(got[True][n], got[False][n]), n
    a, b = ops.gemm(x.to(BF), w.to(BF)), ops.gemm(x.to(BF), w2.to(BF))
    wants = {"plain": a, "pair0": a, "pair1": b, "batch0": a, "batch1": b, "swiglu": ops.swiglu(a, b)}
    wants |= {n: ops.gemm(xq, wq, scale_a=xs, scale_w=ws) for n in f8}
    for n, want in wants.items():
        assert ops.max_rel_err(got[True][n], want) < 1e-2, n
