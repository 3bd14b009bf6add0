"""The tensor-core GEMM with tokens as the MMA's A operand, at the edges of its tiles: token groups of 8 ... 512 rows, ragged
N, plain / bias / GELU / residual / SwiGLU epilogues, packed and row-major operands; one to ten K runs in one CTA and over
clusters of 2 to 8."""
from __future__ import annotations

import pytest
import torch

from aginfer_b200.recipes import Tensor, U32, Weight
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


def quantised(x):
    q, s = ops.quantize_e4m3(x)
    return q, s.reshape(())


@pytest.mark.parametrize("M,N,K,runs,ranks", [
    (70, 272, 5120, 10, 1), (70, 272, 5120, 10, 2), (70, 272, 5120, 10, 3), (77, 256, 5120, 10, 5), (72, 256, 5120, 10, 8),
    (130, 144, 1536, 3, 1), (130, 144, 1536, 3, 2), (130, 144, 1536, 3, 3), (33, 160, 3072, 6, 6), (33, 160, 3072, 6, 4),
    (257, 80, 1792, 7, 4), (257, 80, 1792, 7, 6), (129, 48, 1664, 4, 4), (129, 48, 1664, 4, 1), (96, 1536, 1536, 6, 3),
    (96, 1536, 1536, 6, 2), (513, 2048, 1536, 3, 3), (513, 2048, 1536, 3, 1), (600, 1536, 1024, 2, 2), (450, 3584, 1536, 3, 3)])
@pytest.mark.parametrize("kind", ["bf16", "e4m3", "packed"])
def test_the_sum_over_k_does_not_depend_on_the_cluster(tmp_path, kind, M, N, K, runs, ranks):
    """K in 3 to 10 runs, kept by one CTA or shared by 2 to 8 ranks that hold one run, several, or unequal counts: the
    same bits as one CTA that adds all of them, and the oracle's values."""
    from aginfer_b200.recipes.builder import FLAG_BIAS, FLAG_SCALED, TK_CLUSTERS, tk_tiling

    packed, elem = kind == "packed", 2 if kind == "bf16" else 1
    family = "agi_gemm_tcpk_e4m3" if packed else f"agi_gemm_tk_{kind}"
    if ranks not in TK_CLUSTERS[family]:
        pytest.skip("no such cluster for this type")
    g = torch.Generator().manual_seed(K + M)
    x, wf, bias = torch.randn(M, K, generator=g).to(BF), torch.randn(N, K, generator=g).to(BF), torch.randn(N, generator=g).to(BF)
    if kind == "bf16":
        weights, want = {"w": wf, "b": bias}, ops.gemm(x, wf, bias=bias)
    else:
        (xq, xs), (wq, ws) = quantised(x), quantised(wf)
        weights = {"w": pack_kblock_swizzled(wq) if packed else wq, "b": bias, "s": ws}
        want = ops.gemm(xq, wq, scale_a=xs, scale_w=ws, bias=bias)

    def body(r):
        src, scale = Tensor("x"), None
        if kind != "bf16":
            src, scale = r.alloc((padded_token_rows(M) if packed else M) * K), r.alloc(4)
            r.quantize_e4m3(Tensor("x"), src, scale, M * K, packed=(M, K) if packed else None)
        for out, C in (("y", ranks), ("one", 1)):
            t = tk_tiling(M, (N,), K, elem, runs=runs, clusters=(C,))
            assert t["C"] == C and t["runs"] == runs
            r._gemm_tk(family, "gemm", t, src, [(Weight("w"), Weight("b"), Weight("s") if scale else None, Tensor(out), N, N)],
                       M, K, padded_token_rows(M) if packed else K, FLAG_BIAS | (FLAG_SCALED if scale else 0), scale_a=scale)
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, weights, {"x": x}, {"y": (BF, (M, N)), "one": (BF, (M, N)), "status": (torch.int32, (1,))}, body,
                        repeats=2)
    assert got["status"].item() == 0, hex(got["status"].item())
    assert torch.equal(got["y"], got["one"])
    assert ops.max_rel_err(got["y"], want) < 1e-2


@pytest.mark.parametrize("kind,M,I,K,bias,runs", [
    ("e4m3", 77, 96, 256, False, 1), ("e4m3", 101, 272, 2048, True, 2), ("e4m3", 288, 3456, 1280, True, 1),
    ("packed", 77, 256, 256, True, 1), ("packed", 130, 144, 1536, False, 3), ("packed", 288, 1408, 2048, False, 1),
    ("bf16", 70, 96, 128, True, 1), ("bf16", 129, 1000, 1024, False, 2), ("bf16", 50, 384, 1024, True, None),
    ("bf16", 17, 4096, 1024, False, None), ("e4m3", 300, 130, 256, True, 1)])
def test_gemm_swiglu_matches_separate_launches(tmp_path, kind, M, I, K, bias, runs):
    """SwiGLU in the epilogue, as one launch over gate and up and as two (the up product times silu of the stored gate):
    with K summed alike, the same bits, the same maximum and the same quantisation as two products and the elementwise
    kernels.  Up to 64 tokens in bf16 K is cut over a cluster as the tile asks, so there the oracle decides alone."""
    g = torch.Generator().manual_seed(I + K + M)
    x = torch.randn(M, K, generator=g).to(BF)
    dtype, packed = ("bf16" if kind == "bf16" else "e4m3"), kind == "packed"
    weights, products = {}, []
    xq, xs = quantised(x)
    for name in ("gate", "up"):
        wf, b = (torch.randn(I, K, generator=g) * 0.05).to(BF), (torch.randn(I, generator=g) * 0.5).to(BF)
        kw = dict(bias=b if bias else None)
        if dtype == "bf16":
            weights[name] = wf
            products.append(ops.gemm(x, wf, **kw))
        else:
            wq, ws = quantised(wf)
            weights.update({name: pack_kblock_swizzled(wq) if packed else wq, f"{name}_s": ws})
            products.append(ops.gemm(xq, wq, scale_a=xs, scale_w=ws, **kw))
        if bias:
            weights[f"{name}_b"] = b
    want = ops.swiglu(*products)
    names = ["fused", "split", "plain"] if runs is not None else ["fused", "plain"]
    cols = -(-I // 8) * 8                                # the elementwise kernel works on whole vectors

    def body(r):
        src, scale = Tensor("x"), None
        if dtype == "e4m3":
            src, scale = r.alloc((padded_token_rows(M) if packed else M) * K), r.alloc(4)
            r.quantize_e4m3(Tensor("x"), src, scale, M * K, packed=(M, K) if packed else None)
        part = lambda n: (Weight(n), Weight(f"{n}_b") if bias else None, Weight(f"{n}_s") if scale else None)
        kw = dict(dtype=dtype, scale_a=scale, packed=packed, runs=runs)
        for name in names:
            out = Tensor(name)
            if name == "plain":
                gate, up, amax = r.alloc(M * cols * 2), r.alloc(M * cols * 2), None
                r.gemm_group(src, [(*part("gate"), gate, I, cols), (*part("up"), up, I, cols)], M, K, **kw)
                if cols == I:
                    r.swiglu(gate, up, out, M, I, I)
                else:
                    wide = r.alloc(M * cols * 2)
                    r.swiglu(gate, up, wide, M, cols, cols)
                    r.launch("agi_copy_rows_bf16", (64, 1, 1), (256, 1, 1), [wide, out, U32(M), U32(I), U32(cols), U32(I)])
            else:
                amax = r.counter()
                r.gemm_swiglu(src, part("gate"), part("up"), out, M, I, K, amax=amax,
                              scratch=r.alloc(M * I * 2) if name == "split" else None, **kw)
            r.quantize_e4m3(out, Tensor(f"{name}_q"), Tensor(f"{name}_scale"), M * I, amax=amax)
        r.export_status(Tensor("status"))

    outputs = {"status": (torch.int32, (1,))}
    for name in names:
        outputs.update({name: (BF, (M, I)), f"{name}_q": (torch.uint8, (M, I)), f"{name}_scale": (torch.float32, (1,))})
    got, _ = run_recipe(tmp_path, weights, {"x": x}, outputs, body, repeats=2)
    assert got["status"].item() == 0, hex(got["status"].item())
    for name in names:
        # gate, up and result each within one bf16 step (2^-7 at most) where an fp32 sum in another order rounds away
        assert ops.max_rel_err(got[name], want) < 3 * 2.0 ** -7, name
        if runs is not None:
            for what in ("", "_q", "_scale"):
                assert torch.equal(got[name + what], got["plain" + what]), (name, what)
        amax = got[name].float().abs().max()
        assert got[f"{name}_scale"].item() == pytest.approx((amax / 448).item(), rel=1e-6)
