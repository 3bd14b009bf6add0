"""Parity of each kernel family with the CPU oracle, launched through the packaged recipe path:
modelc compile -> AIM -> C ABI loader -> cuLaunchKernel from the CUBIN."""
from __future__ import annotations

import pytest
import torch

from aginfer_b200.recipes import Tensor, Weight
from oracle import ops
from tests.gpu_util import MAX_REL, run_recipe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def randn(*shape, seed=0, std=1.0, dtype=BF):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * std).to(dtype)


def test_vector_add_through_the_whole_pipeline(tmp_path):
    # the reference's own GPU test (tests/cuda_runtime_test.cc:50-76): 16 floats, exact to 1e-6
    left = torch.arange(16, dtype=torch.float32) * 0.5
    right = torch.arange(16, dtype=torch.float32) * -0.25
    got, stats = run_recipe(tmp_path, {}, {"left": left, "right": right}, {"output": (torch.float32, (16,))},
                            lambda r: r.vector_add(Tensor("left"), Tensor("right"), Tensor("output"), 16), repeats=3)
    assert torch.allclose(got["output"], left + right, atol=1e-6)
    assert stats["enqueues"] == 3 and stats["graph_launches"] == 3 and stats["graphs_built"] == 1
    assert stats["kernel_launches"] == stats["launches_per_enqueue"] == 2  # prologue + kernel, captured once


def test_plain_launch_mode_matches_graph_mode(tmp_path):
    from aginfer_b200.runtime import NO_GRAPH_REPLAY
    left, right = torch.ones(16), torch.full((16,), 2.0)
    got, stats = run_recipe(tmp_path, {}, {"left": left, "right": right}, {"output": (torch.float32, (16,))},
                            lambda r: r.vector_add(Tensor("left"), Tensor("right"), Tensor("output"), 16),
                            flags=NO_GRAPH_REPLAY, repeats=2)
    assert torch.equal(got["output"], torch.full((16,), 3.0))
    assert stats["graph_launches"] == 0 and stats["kernel_launches"] == 4


@pytest.mark.parametrize("shape", [(1, 2048), (17, 1536), (288, 2048), (3, 1000), (1024, 11008)])
def test_quantize_e4m3_is_bit_exact(tmp_path, shape):
    x = randn(*shape, seed=1)
    want_q, want_s = ops.quantize_e4m3(x)
    n = x.numel()

    def body(r):
        r.quantize_e4m3(Tensor("x"), Tensor("q"), Tensor("scale"), n)

    got, _ = run_recipe(tmp_path, {}, {"x": x}, {"q": (torch.float8_e4m3fn, shape), "scale": (torch.float32, (1,))},
                        body, repeats=2)
    assert got["scale"].view(torch.int32).item() == want_s.view(torch.int32).item()
    assert torch.equal(got["q"].view(torch.uint8), want_q.view(torch.uint8))


def test_quantize_all_zero_input(tmp_path):
    x = torch.zeros(4, 64, dtype=BF)
    got, _ = run_recipe(tmp_path, {}, {"x": x}, {"q": (torch.float8_e4m3fn, (4, 64)), "scale": (torch.float32, (1,))},
                        lambda r: r.quantize_e4m3(Tensor("x"), Tensor("q"), Tensor("scale"), 256))
    assert got["scale"].item() == 1.0 and int(got["q"].view(torch.uint8).max()) == 0


@pytest.mark.parametrize("rows,cols", [(288, 2048), (17, 1536), (5, 1280), (2, 3584)])
def test_rmsnorm(tmp_path, rows, cols):
    x, gain = randn(rows, cols, seed=2), (1 + randn(cols, seed=3, std=0.1).float()).to(BF)
    got, _ = run_recipe(tmp_path, {"norm.weight": gain}, {"x": x}, {"y": (BF, (rows, cols))},
                        lambda r: r.rmsnorm(Tensor("x"), Weight("norm.weight"), Tensor("y"), rows, cols, 1e-6))
    assert ops.max_rel_err(got["y"], ops.rmsnorm(x, gain, 1e-6)) < 1e-2


@pytest.mark.parametrize("modulated", [False, True])
def test_layernorm_and_adaln_modulation(tmp_path, modulated):
    rows, cols = 17, 1536
    x = (randn(rows, cols, seed=4).float() * 3 + 1.5).to(BF)
    mod = randn(2 * cols, seed=5, std=0.3)

    def body(r):
        if modulated:
            r.layernorm(Tensor("x"), Tensor("y"), rows, cols, 1e-5, scale=Weight("mod"), shift=Weight("mod") + 2 * cols)
        else:
            r.layernorm(Tensor("x"), Tensor("y"), rows, cols, 1e-5)

    got, _ = run_recipe(tmp_path, {"mod": mod}, {"x": x}, {"y": (BF, (rows, cols))}, body)
    want = ops.layernorm(x, 1e-5, mod[:cols], mod[cols:]) if modulated else ops.layernorm(x, 1e-5)
    assert ops.max_rel_err(got["y"], want) < 1e-2


@pytest.mark.parametrize("rows,cols", [(17, 1536), (50, 1536), (3, 8), (5, 8192), (2, 8200)])
def test_layernorm_that_fetches_its_modulation_early(tmp_path, rows, cols):
    """Scale and shift written by the profile itself, then read ahead of the dependency wait behind a launch that
    releases its successors only after its own wait: the values of the ordinary order, bit for bit, under programmatic
    dependent launch, for rows that stay in registers and rows that do not."""
    from aginfer_b200 import runtime as rt
    from aginfer_b200.recipes import U32
    x, mod = (randn(rows, cols, seed=4).float() * 3 + 1.5).to(BF), randn(2, cols, seed=5, std=0.3)

    def body(r):
        held, ones, late = r.alloc(4 * cols), r.alloc(2 * rows * cols), r.alloc(4 * cols)
        copy = lambda src, dst, n: r.launch("agi_copy_rows_bf16", (64, 1, 1), (256, 1, 1),
                                            [src, dst, U32(n // cols), U32(cols), U32(cols), U32(cols)])
        copy(Tensor("mod"), held, 2 * cols)
        copy(Tensor("x"), ones, rows * cols)
        # x + 0: the launch between the modulation's writer and its early reader
        r.launch("agi_add_rows_bf16", (64, 1, 1), (256, 1, 1), [ones, late, U32(rows), U32(cols), U32(cols), U32(1)])
        for out, static in (("early", True), ("plain", False)):
            r.layernorm(ones, Tensor(out), rows, cols, 1e-5, scale=held, shift=held + 2 * cols, static_modulation=static)

    got, _ = run_recipe(tmp_path, {}, {"x": x, "mod": mod}, {"early": (BF, (rows, cols)), "plain": (BF, (rows, cols))}, body,
                        flags=rt.PROGRAMMATIC_LAUNCH, repeats=3)
    assert torch.equal(got["early"], got["plain"])
    assert ops.max_rel_err(got["early"], ops.layernorm(x, 1e-5, mod[0], mod[1])) < 1e-2


def test_rope_1d(tmp_path):
    rows, heads, d = 288, 18, 128  # 16 query + 2 key heads rotated, 2 value heads untouched
    x = randn(rows, (heads + 2) * d, seed=6)
    from aginfer_b200.recipes import U32
    width = x.shape[1]

    def body(r):
        r.launch("agi_copy_rows_bf16", (592, 1, 1), (256, 1, 1),
                 [Tensor("x"), Tensor("y"), U32(rows), U32(width), U32(width), U32(width)])
        r.rope(Tensor("y"), rows, heads, d, width, 1e6)

    got, _ = run_recipe(tmp_path, {}, {"x": x}, {"y": (BF, x.shape)}, body)
    want = x.clone().view(rows, heads + 2, d)
    want[:, :heads] = ops.rope(want[:, :heads], 1e6)
    assert torch.equal(got["y"].view(rows, heads + 2, d)[:, heads:], x.view(rows, heads + 2, d)[:, heads:])
    assert ops.max_rel_err(got["y"], want.view(rows, -1)) < 1e-2


def test_rope_over_two_tensors_in_one_launch_matches_two_launches(tmp_path):
    rows, hq, hk, d, offset = 50, 8, 4, 128, 88    # the action expert's queries and new keys
    q, k = randn(rows, hq * d, seed=7), randn(rows, hk * d, seed=8)
    from aginfer_b200.recipes import U32

    def body(r):
        for src, dst, width in (("q", "q1", hq * d), ("q", "q2", hq * d), ("k", "k1", hk * d), ("k", "k2", hk * d)):
            r.launch("agi_copy_rows_bf16", (200, 1, 1), (256, 1, 1),
                     [Tensor(src), Tensor(dst), U32(rows), U32(width), U32(width), U32(width)])
        r.rope(Tensor("q1"), rows, hq, d, hq * d, 1e6, pos_offset=offset)
        r.rope(Tensor("k1"), rows, hk, d, hk * d, 1e6, pos_offset=offset)
        r.rope_pair(Tensor("q2"), hq, hq * d, Tensor("k2"), hk, hk * d, rows, d, 1e6, pos_offset=offset)

    got, _ = run_recipe(tmp_path, {}, {"q": q, "k": k}, {"q1": (BF, q.shape), "q2": (BF, q.shape), "k1": (BF, k.shape),
                                                         "k2": (BF, k.shape)}, body)
    # two compilations of the same arithmetic may contract multiply-adds differently: equal to rounding, not bit for bit
    assert ops.max_rel_err(got["q2"], got["q1"].float()) < 5e-3 and ops.max_rel_err(got["k2"], got["k1"].float()) < 5e-3
    assert ops.max_rel_err(got["q2"], ops.rope(q.view(rows, hq, d), 1e6, offset).reshape(rows, -1)) < 1e-2
    assert ops.max_rel_err(got["k2"], ops.rope(k.view(rows, hk, d), 1e6, offset).reshape(rows, -1)) < 1e-2


def test_mrope_sections(tmp_path):
    from aginfer_b200.recipes import U32
    rows, heads, d = 64, 4, 128
    x = randn(rows, heads * d, seed=7)
    g = torch.Generator().manual_seed(8)
    pos = torch.randint(0, 300, (3, rows), generator=g, dtype=torch.int32)

    def body(r):
        r.launch("agi_copy_rows_bf16", (128, 1, 1), (256, 1, 1),
                 [Tensor("x"), Tensor("y"), U32(rows), U32(heads * d), U32(heads * d), U32(heads * d)])
        r.mrope(Tensor("y"), Tensor("pos"), rows, heads, d, heads * d, 1e6, (16, 24, 24))

    got, _ = run_recipe(tmp_path, {}, {"x": x, "pos": pos}, {"y": (BF, x.shape)}, body)
    want = ops.mrope(x.view(rows, heads, d), pos, 1e6, (16, 24, 24)).view(rows, -1)
    assert ops.max_rel_err(got["y"], want) < 1e-2


ATTENTION_CASES = [
    # q_rows, kv_rows, q_heads, kv_heads, head_dim, mask, mask_arg
    (288, 288, 16, 2, 128, "causal", 0),      # decoder layer, GQA causal
    (17, 17, 32, 32, 48, "none", 0),          # DiT self attention
    (17, 300, 32, 32, 48, "none", 0),         # DiT cross attention
    (512, 512, 16, 16, 80, "block", 64),      # vision window attention
    (512, 512, 16, 16, 80, "block", 256),     # vision full attention, per image
    (50, 306, 8, 4, 128, "causal", 256),      # action expert over [prefix | suffix]
    (5, 3, 2, 1, 16, "none", 0),              # ragged, smaller than one tile
    (32, 77, 6, 3, 64, "causal", 45),         # few queries, GQA, causal with an offset
    (20, 40, 4, 4, 32, "block", 10),          # few queries, block-diagonal
]


@pytest.mark.parametrize("algorithm", ["warp_per_row", "keys_in_smem", "key_split", "auto"])
@pytest.mark.parametrize("case", ATTENTION_CASES, ids=lambda c: "x".join(map(str, c)))
def test_attention(tmp_path, case, algorithm):
    sq, skv, hq, hkv, d, mask, arg = case
    q, k, v = randn(sq, hq * d, seed=9), randn(skv, hkv * d, seed=10), randn(skv, hkv * d, seed=11)
    got, _ = run_recipe(tmp_path, {}, {"q": q, "k": k, "v": v}, {"o": (BF, (sq, hq * d))}, lambda r: r.attention(
        Tensor("q"), Tensor("k"), Tensor("v"), Tensor("o"), q_rows=sq, kv_rows=skv, q_heads=hq, kv_heads=hkv,
        head_dim=d, q_stride=hq * d, k_stride=hkv * d, v_stride=hkv * d, o_stride=hq * d, mask=mask, mask_arg=arg,
        algorithm=algorithm))
    want = ops.attention(q.view(sq, hq, d), k.view(skv, hkv, d), v.view(skv, hkv, d), mask=mask, mask_arg=arg)
    assert ops.max_rel_err(got["o"], want.reshape(sq, -1)) < MAX_REL


@pytest.mark.parametrize("case,static_rows", [((17, 300, 32, 32, 48, "none", 0), None), ((50, 306, 8, 4, 128, "causal", 256), 256),
                                              ((50, 306, 8, 4, 128, "none", 0), 250), ((64, 40, 4, 2, 96, "none", 0), 16),
                                              ((17, 17, 32, 32, 48, "none", 0), 5)], ids=lambda c: str(c).replace(" ", ""))
def test_attention_with_keys_requested_ahead_of_the_dependency_wait(tmp_path, case, static_rows):
    """Few query rows, keys / values (or a leading part of them) declared static: the kernel requests those rows before
    its grid-dependency wait.  Here they are profile inputs, so any split must give the result of the plain call."""
    sq, skv, hq, hkv, d, mask, arg = case
    q, k, v = randn(sq, hq * d, seed=9), randn(skv, hkv * d, seed=10), randn(skv, hkv * d, seed=11)

    def body(r):
        for name, kw in (("o_plain", {}), ("o_early", {"kv_static": True, "kv_static_rows": static_rows})):
            r.attention(Tensor("q"), Tensor("k"), Tensor("v"), Tensor(name), q_rows=sq, kv_rows=skv, q_heads=hq, kv_heads=hkv,
                        head_dim=d, q_stride=hq * d, k_stride=hkv * d, v_stride=hkv * d, o_stride=hq * d, mask=mask,
                        mask_arg=arg, **kw)

    got, _ = run_recipe(tmp_path, {}, {"q": q, "k": k, "v": v}, {"o_plain": (BF, (sq, hq * d)), "o_early": (BF, (sq, hq * d))}, body)
    want = ops.attention(q.view(sq, hq, d), k.view(skv, hkv, d), v.view(skv, hkv, d), mask=mask, mask_arg=arg)
    assert torch.equal(got["o_plain"], got["o_early"])
    assert ops.max_rel_err(got["o_early"], want.reshape(sq, -1)) < MAX_REL


FEW_ROW_CASES = [
    # at most 32 keys and heads up to 64 wide: the split by value columns; otherwise the split by keys
    (17, 17, 4, 4, 48, "causal", 0),
    (24, 30, 4, 2, 64, "causal", 6),
    (20, 20, 4, 4, 32, "block", 7),
    (30, 20, 2, 2, 48, "block", 10),                     # rows 20 - 29: their block begins behind the last key
    (64, 33, 2, 1, 16, "block", 11),                     # the same, keys split
    (50, 70, 4, 2, 128, "block", 33),                    # wide heads, last block cut by the keys
    (50, 40, 2, 2, 96, "block", 45),                     # ... and a row block of which some rows see keys and some none
    (17, 30, 2, 2, 48, "causal", 2 ** 32 - 17),          # the last row's offset is the largest 32-bit number: every key
    (33, 70, 2, 1, 64, "causal", 2 ** 32 - 33),
    (20, 40, 2, 1, 128, "causal", 2 ** 32 - 20),
]


@pytest.mark.parametrize("case", FEW_ROW_CASES, ids=lambda c: "x".join(map(str, c)))
def test_attention_of_few_rows_sees_the_masks_keys(tmp_path, case):
    sq, skv, hq, hkv, d, mask, arg = case
    q, k, v = randn(sq, hq * d, seed=9), randn(skv, hkv * d, seed=10), randn(skv, hkv * d, seed=11)

    def body(r):
        r.attention(Tensor("q"), Tensor("k"), Tensor("v"), Tensor("o"), q_rows=sq, kv_rows=skv, q_heads=hq, kv_heads=hkv,
                    head_dim=d, q_stride=hq * d, k_stride=hkv * d, v_stride=hkv * d, o_stride=hq * d, mask=mask, mask_arg=arg,
                    algorithm="mma")
        assert r.profiles[0].launches[-1]["kernel"].startswith("agi_attention_mma_bf16")

    got, _ = run_recipe(tmp_path, {}, {"q": q, "k": k, "v": v}, {"o": (BF, (sq, hq * d))}, body)
    want = ops.attention(q.view(sq, hq, d), k.view(skv, hkv, d), v.view(skv, hkv, d), mask=mask, mask_arg=arg)
    assert ops.max_rel_err(got["o"], want.nan_to_num(0.0).reshape(sq, -1)) < MAX_REL      # no visible key: zeros


FA_CASES = [
    (288, 288, 16, 2, 128, "causal", 0),     # decoder prefill: grouped-query, 4.5 key tiles
    (512, 512, 16, 16, 80, "block", 64),     # vision windows
    (512, 512, 16, 16, 80, "block", 256),    # vision full-attention layers: one block per image
    (100, 300, 4, 4, 64, "none", 0),         # cross attention, ragged both ways
    (70, 130, 6, 3, 48, "causal", 60),       # queries are the last 70 of 130 positions
    (17, 300, 32, 32, 48, "none", 0),        # fewer rows than one block
    (200, 200, 2, 1, 128, "block", 24),      # blocks that straddle key tiles and row blocks
]


@pytest.mark.parametrize("case", FA_CASES, ids=lambda c: "x".join(map(str, c)))
def test_attention_streaming_mma(tmp_path, case):
    sq, skv, hq, hkv, d, mask, arg = case
    q, k, v = randn(sq, hq * d, seed=9), randn(skv, hkv * d, seed=10), randn(skv, hkv * d, seed=11)
    got, _ = run_recipe(tmp_path, {}, {"q": q, "k": k, "v": v}, {"o": (BF, (sq, hq * d))}, lambda r: r.attention(
        Tensor("q"), Tensor("k"), Tensor("v"), Tensor("o"), q_rows=sq, kv_rows=skv, q_heads=hq, kv_heads=hkv,
        head_dim=d, q_stride=hq * d, k_stride=hkv * d, v_stride=hkv * d, o_stride=hq * d, mask=mask, mask_arg=arg,
        algorithm="fa"))
    want = ops.attention(q.view(sq, hq, d), k.view(skv, hkv, d), v.view(skv, hkv, d), mask=mask, mask_arg=arg)
    assert ops.max_rel_err(got["o"], want.reshape(sq, -1)) < MAX_REL


def test_swiglu(tmp_path):
    rows, inter = 33, 11008
    gu = randn(rows, 2 * inter, seed=12)
    got, _ = run_recipe(tmp_path, {}, {"gu": gu}, {"h": (BF, (rows, inter))}, lambda r: r.swiglu(
        Tensor("gu"), Tensor("gu"), Tensor("h"), rows, inter, 2 * inter))
    # gate == up pointer here (same column block); the strided form is covered by the layer test
    assert ops.max_rel_err(got["h"], ops.swiglu(gu[:, :inter], gu[:, :inter])) < 1e-2


@pytest.mark.parametrize("M,N,K", [(17, 1536, 1536), (288, 2560, 2048), (1, 64, 96), (70, 100, 40)])
def test_gemm_simt_bf16(tmp_path, M, N, K):
    x, w = randn(M, K, seed=13), randn(N, K, seed=14, std=0.02)
    bias, res = randn(N, seed=15, std=0.1), randn(M, N, seed=16)
    got, _ = run_recipe(tmp_path, {"w": w, "b": bias}, {"x": x, "res": res}, {"y": (BF, (M, N))}, lambda r: r.gemm(
        Tensor("x"), Weight("w"), Tensor("y"), M, N, K, bias=Weight("b"), residual=Tensor("res"), act="gelu_tanh"))
    want = ops.gemm(x, w, bias=bias, residual=res, act="gelu_tanh")
    assert ops.max_rel_err(got["y"], want) < MAX_REL


def test_gemm_simt_e4m3_scaled(tmp_path):
    M, N, K = 16, 2048, 2048
    x, wf = randn(M, K, seed=1), randn(N, K, seed=17, std=0.02)
    wq, ws = ops.quantize_e4m3(wf)
    xq, xs = ops.quantize_e4m3(x)

    def body(r):
        q, s = r.alloc(M * K), r.alloc(4)
        r.quantize_e4m3(Tensor("x"), q, s, M * K)
        r.gemm(q, Weight("w"), Tensor("y"), M, N, K, dtype="e4m3", scale_a=s, scale_w=Weight("w_scale"))

    got, _ = run_recipe(tmp_path, {"w": wq, "w_scale": ws.reshape(())}, {"x": x}, {"y": (BF, (M, N))}, body)
    want = ops.gemm(xq, wq, scale_a=xs, scale_w=ws)
    assert ops.max_rel_err(got["y"], want) < 1e-2
    # and the quantised product stays close to the unquantised one
    assert ops.max_rel_err(got["y"], ops.gemm(x, wf.to(BF))) < 0.1


TC_CASES = [
    # M, N, K, dtype, splits (None = builder's choice), epilogue
    (17, 1536, 1536, "bf16", None, "plain"),       # DiT projection, split-K 12
    (17, 1536, 1536, "bf16", 1, "bias_gelu_res"),  # same, one slice, full epilogue
    (17, 6144, 1536, "bf16", None, "bias_gelu"),   # DiT MLP up
    (17, 1536, 6144, "bf16", None, "bias_res"),    # DiT MLP down
    (288, 2560, 2048, "bf16", None, "bias"),       # decoder QKV, two token tiles of 144
    (288, 2048, 11008, "bf16", None, "res"),       # decoder down projection
    (50, 1024, 4096, "bf16", None, "plain"),       # action expert
    (1, 2048, 2048, "e4m3", None, "plain"),        # FP8 sweep corners
    (16, 11008, 2048, "e4m3", None, "plain"),
    (64, 2048, 11008, "e4m3", None, "plain"),
    (288, 2560, 2048, "e4m3", None, "bias"),
    (1024, 1536, 1536, "e4m3", None, "plain"),
    (300, 1000, 512, "bf16", None, "bias"),        # ragged: N and M not multiples of the tile
    (5, 130, 128, "e4m3", 1, "plain"),
]


@pytest.mark.parametrize("case", TC_CASES, ids=lambda c: "-".join(map(str, c)))
def test_gemm_tcgen05(tmp_path, case):
    M, N, K, dtype, splits, epi = case
    x, wf = randn(M, K, seed=21), randn(N, K, seed=22, std=0.02)
    bias = randn(N, seed=23, std=0.1) if "bias" in epi else None
    res = randn(M, N, seed=24) if "res" in epi else None
    act = "gelu_tanh" if "gelu" in epi else None
    weights, inputs = {}, {"x": x}
    if dtype == "e4m3":
        wq, ws = ops.quantize_e4m3(wf)
        xq, xs = ops.quantize_e4m3(x)
        weights.update({"w": wq, "w_scale": ws.reshape(())})
        want = ops.gemm(xq, wq, bias=bias, residual=res, act=act, scale_a=xs, scale_w=ws)
    else:
        weights["w"] = wf.to(BF)
        want = ops.gemm(x, wf.to(BF), bias=bias, residual=res, act=act)
    if bias is not None:
        weights["b"] = bias
    if res is not None:
        inputs["res"] = res

    def body(r):
        kw = dict(bias=Weight("b") if bias is not None else None, residual=Tensor("res") if res is not None else None,
                  act=act, tactic="tcgen05", splits=splits)
        if dtype == "e4m3":
            q, s = r.alloc(M * K), r.alloc(4)
            r.quantize_e4m3(Tensor("x"), q, s, M * K)
            r.gemm(q, Weight("w"), Tensor("y"), M, N, K, dtype="e4m3", scale_a=s, scale_w=Weight("w_scale"), **kw)
        else:
            r.gemm(Tensor("x"), Weight("w"), Tensor("y"), M, N, K, **kw)
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, weights, inputs, {"y": (BF, (M, N)), "status": (torch.int32, (1,))}, body, repeats=3)
    assert got["status"].item() == 0, hex(got["status"].item())
    err = ops.max_rel_err(got["y"], want)
    assert err < (1e-2 if dtype == "bf16" else 1e-2), err


WIDE_CASES = [
    (1024, 11008, 2048, "e4m3", 1, "plain"),        # prefill gate/up: 43 x 4 tiles of 256 x 256
    (1024, 2048, 11008, "bf16", 4, "res"),          # prefill down projection, K in four slices
    (288, 2560, 2048, "bf16", 1, "bias_gelu"),      # two token tiles of 144
    (300, 1000, 512, "bf16", 2, "bias_res"),        # ragged: N, M not multiples of the tile; two slices
    (130, 300, 256, "e4m3", 1, "bias"),             # second 128-row half mostly past N
    (128, 256, 128, "bf16", 1, "plain"),            # one K block
]


@pytest.mark.parametrize("case", WIDE_CASES, ids=lambda c: "-".join(map(str, c)))
def test_gemm_tcgen05_wide(tmp_path, case):
    """256-row tensor-core kernel (two accumulators in tensor memory), direct and split-K epilogues."""
    M, N, K, dtype, splits, epi = case
    x, wf = randn(M, K, seed=41), randn(N, K, seed=42, std=0.02)
    bias = randn(N, seed=43, std=0.1) if "bias" in epi else None
    res = randn(M, N, seed=44) if "res" in epi else None
    act = "gelu_tanh" if "gelu" in epi else None
    weights, inputs = {}, {"x": x}
    if dtype == "e4m3":
        wq, ws = ops.quantize_e4m3(wf)
        xq, xs = ops.quantize_e4m3(x)
        weights.update({"w": wq, "w_scale": ws.reshape(())})
        want = ops.gemm(xq, wq, bias=bias, residual=res, act=act, scale_a=xs, scale_w=ws)
    else:
        weights["w"] = wf.to(BF)
        want = ops.gemm(x, wf.to(BF), bias=bias, residual=res, act=act)
    if bias is not None:
        weights["b"] = bias
    if res is not None:
        inputs["res"] = res

    def body(r):
        kw = dict(bias=Weight("b") if bias is not None else None, residual=Tensor("res") if res is not None else None,
                  act=act, tactic="tcgen05_wide", splits=splits)
        if dtype == "e4m3":
            q, s = r.alloc(M * K), r.alloc(4)
            r.quantize_e4m3(Tensor("x"), q, s, M * K)
            r.gemm(q, Weight("w"), Tensor("y"), M, N, K, dtype="e4m3", scale_a=s, scale_w=Weight("w_scale"), **kw)
        else:
            r.gemm(Tensor("x"), Weight("w"), Tensor("y"), M, N, K, **kw)
        r.export_status(Tensor("status"))

    got, recipe = run_recipe(tmp_path, weights, inputs, {"y": (BF, (M, N)), "status": (torch.int32, (1,))}, body,
                             repeats=3)
    assert got["status"].item() == 0, hex(got["status"].item())
    assert ops.max_rel_err(got["y"], want) < 1e-2


@pytest.mark.parametrize("dtype,M,K,widths", [("e4m3", 288, 2048, (2048, 256, 256)), ("bf16", 300, 512, (1000, 72)),
                                              # up to 64 tokens in bf16: K slices of every tile in a cluster (c8, c2, c4)
                                              ("bf16", 50, 1024, (1024, 512, 512)), ("bf16", 50, 1024, (4096, 4096)),
                                              ("bf16", 17, 1536, (1536, 1000, 520)),
                                              ("e4m3", 512, 1280, (3456, 3456)), ("bf16", 17, 128, (128,))])
def test_gemm_group(tmp_path, dtype, M, K, widths):
    """Q | K | V style: several weight matrices over one activation matrix in one tensor-core launch."""
    x = randn(M, K, seed=61)
    weights, wants, outs = {}, [], {}
    if dtype == "e4m3":
        xq, xs = ops.quantize_e4m3(x)
    for i, n in enumerate(widths):
        wf, bias = randn(n, K, seed=62 + i, std=0.02), randn(n, seed=72 + i, std=0.1)
        weights[f"b{i}"] = bias
        if dtype == "e4m3":
            wq, ws = ops.quantize_e4m3(wf)
            weights[f"w{i}"], weights[f"s{i}"] = wq, ws.reshape(())
            wants.append(ops.gemm(xq, wq, bias=bias, scale_a=xs, scale_w=ws))
        else:
            weights[f"w{i}"] = wf.to(BF)
            wants.append(ops.gemm(x, wf.to(BF), bias=bias))
        outs[f"y{i}"] = (BF, (M, n))

    def body(r):
        src, scale = Tensor("x"), None
        if dtype == "e4m3":
            src, scale = r.alloc(M * K), r.alloc(4)
            r.quantize_e4m3(Tensor("x"), src, scale, M * K)
        r.gemm_group(src, [(Weight(f"w{i}"), Weight(f"b{i}"), Weight(f"s{i}") if dtype == "e4m3" else None,
                            Tensor(f"y{i}"), n, n) for i, n in enumerate(widths)], M, K, dtype=dtype, scale_a=scale)
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, weights, {"x": x}, {**outs, "status": (torch.int32, (1,))}, body, repeats=2)
    assert got["status"].item() == 0
    for i, want in enumerate(wants):
        assert ops.max_rel_err(got[f"y{i}"], want) < 1e-2, i


def test_producers_that_fold_the_amax_match_the_separate_pass(tmp_path):
    """RMSNorm / SwiGLU variants that leave max |y| behind: the quantisation that follows must produce the same
    bytes and the same scale as the two-pass form (bit-exact tier)."""
    rows, cols = 288, 2048
    x, gain = randn(rows, cols, seed=81), (1.0 + 0.1 * randn(cols, seed=82).float()).to(BF)
    gu = randn(rows, 2 * cols, seed=83)

    def body(r):
        y1, y2, a, h1, h2 = (r.alloc(rows * cols * 2) for _ in range(5))
        amax = r.counter()
        r.rmsnorm(Tensor("x"), Weight("gain"), y1, rows, cols, 1e-6)
        r.quantize_e4m3(y1, Tensor("q_two_pass"), Tensor("s_two_pass"), rows * cols)
        r.rmsnorm(Tensor("x"), Weight("gain"), y2, rows, cols, 1e-6, amax=amax)
        r.quantize_e4m3(y2, Tensor("q_folded"), Tensor("s_folded"), rows * cols, amax=amax)
        amax2 = r.counter()
        r.swiglu(Tensor("gu"), Tensor("gu"), h1, rows, cols, 2 * cols)
        r.quantize_e4m3(h1, Tensor("g_two_pass"), Tensor("t_two_pass"), rows * cols)
        r.swiglu(Tensor("gu"), Tensor("gu"), h2, rows, cols, 2 * cols, amax=amax2)
        r.quantize_e4m3(h2, Tensor("g_folded"), Tensor("t_folded"), rows * cols, amax=amax2)

    u8, f32 = (torch.uint8, (rows, cols)), (torch.float32, (1,))
    got, _ = run_recipe(tmp_path, {"gain": gain}, {"x": x, "gu": gu},
                        {"q_two_pass": u8, "s_two_pass": f32, "q_folded": u8, "s_folded": f32, "g_two_pass": u8,
                         "t_two_pass": f32, "g_folded": u8, "t_folded": f32}, body, repeats=2)
    assert torch.equal(got["s_two_pass"], got["s_folded"]) and torch.equal(got["q_two_pass"], got["q_folded"])
    assert torch.equal(got["t_two_pass"], got["t_folded"]) and torch.equal(got["g_two_pass"], got["g_folded"])
    want_q, want_s = ops.quantize_e4m3(ops.rmsnorm(x, gain))
    assert got["s_folded"].item() == pytest.approx(want_s.item(), rel=1e-2)
    assert (got["q_folded"].view(torch.float8_e4m3fn).float() - want_q.float()).abs().max() <= 64   # same grid up to an ulp of y


PACKED_CASES = [(288, 2048, 2048, "bias"), (1024, 11008, 2048, "plain"), (288, 2048, 11008, "res"),
                (130, 300, 256, "bias_gelu"), (512, 1280, 3456, "bias_res"), (17, 128, 128, "plain")]


@pytest.mark.parametrize("tactic", ["auto", "tcgen05_plan"])     # auto may pick the persistent kernel; the plan never does
@pytest.mark.parametrize("case", PACKED_CASES, ids=lambda c: "-".join(map(str, c)))
def test_gemm_packed_operands(tmp_path, case, tactic):
    """Bulk-copy tcgen05 GEMM: weights packed on the CPU (K-block-major, swizzled), activations quantised into
    the same layout on the device; same arithmetic as the row-major kernels."""
    from aginfer_b200.recipes.layout import pack_kblock_swizzled, padded_token_rows
    M, N, K, epi = case
    x, wf = randn(M, K, seed=91), randn(N, K, seed=92, std=0.02)
    bias = randn(N, seed=93, std=0.1) if "bias" in epi else None
    res = randn(M, N, seed=94) if "res" in epi else None
    act = "gelu_tanh" if "gelu" in epi else None
    wq, ws = ops.quantize_e4m3(wf)
    xq, xs = ops.quantize_e4m3(x)
    want = ops.gemm(xq, wq, bias=bias, residual=res, act=act, scale_a=xs, scale_w=ws)
    weights = {"w": pack_kblock_swizzled(wq), "w_scale": ws.reshape(())}
    inputs = {"x": x}
    if bias is not None:
        weights["b"] = bias
    if res is not None:
        inputs["res"] = res

    def body(r):
        q, s = r.alloc(padded_token_rows(M) * K), r.alloc(4)
        r.quantize_e4m3(Tensor("x"), q, s, M * K, packed=(M, K))
        r.gemm(q, Weight("w"), Tensor("y"), M, N, K, dtype="e4m3", scale_a=s, scale_w=Weight("w_scale"),
               bias=Weight("b") if bias is not None else None, residual=Tensor("res") if res is not None else None,
               act=act, packed=True, tactic=tactic)
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, weights, inputs, {"y": (BF, (M, N)), "status": (torch.int32, (1,))}, body, repeats=3)
    assert got["status"].item() == 0, hex(got["status"].item())
    assert ops.max_rel_err(got["y"], want) < 1e-2


def test_gemm_group_packed_operands(tmp_path):
    from aginfer_b200.recipes.layout import pack_kblock_swizzled, padded_token_rows
    M, K, widths = 288, 2048, (2048, 256, 256)
    x = randn(M, K, seed=95)
    xq, xs = ops.quantize_e4m3(x)
    weights, wants = {}, []
    for i, n in enumerate(widths):
        wq, ws = ops.quantize_e4m3(randn(n, K, seed=96 + i, std=0.02))
        bias = randn(n, seed=99 + i, std=0.1)
        weights.update({f"w{i}": pack_kblock_swizzled(wq), f"s{i}": ws.reshape(()), f"b{i}": bias})
        wants.append(ops.gemm(xq, wq, bias=bias, scale_a=xs, scale_w=ws))

    def body(r):
        q, s = r.alloc(padded_token_rows(M) * K), r.alloc(4)
        r.quantize_e4m3(Tensor("x"), q, s, M * K, packed=(M, K))
        r.gemm_group(q, [(Weight(f"w{i}"), Weight(f"b{i}"), Weight(f"s{i}"), Tensor(f"y{i}"), n, n)
                         for i, n in enumerate(widths)], M, K, dtype="e4m3", scale_a=s, packed=True)
        r.export_status(Tensor("status"))

    outs = {f"y{i}": (BF, (M, n)) for i, n in enumerate(widths)}
    got, _ = run_recipe(tmp_path, weights, {"x": x}, {**outs, "status": (torch.int32, (1,))}, body, repeats=2)
    assert got["status"].item() == 0
    for i, want in enumerate(wants):
        assert ops.max_rel_err(got[f"y{i}"], want) < 1e-2, i


@pytest.mark.parametrize("case", [(1024, 11008, 2048, "plain"), (600, 2560, 512, "bias_gelu_res"), (130, 300, 256, "bias"),
                                  (1024, 1536, 1536, "res")], ids=lambda c: "-".join(map(str, c)))
def test_gemm_persistent_packed(tmp_path, case):
    """Persistent tcgen05 kernel (tile loop per CTA, double-buffered accumulators): more tiles than SMs, fewer
    tiles than SMs, ragged edges, every epilogue."""
    from aginfer_b200.recipes.layout import pack_kblock_swizzled, padded_token_rows
    M, N, K, epi = case
    x, wf = randn(M, K, seed=111), randn(N, K, seed=112, std=0.02)
    bias = randn(N, seed=113, std=0.1) if "bias" in epi else None
    res = randn(M, N, seed=114) if "res" in epi else None
    act = "gelu_tanh" if "gelu" in epi else None
    wq, ws = ops.quantize_e4m3(wf)
    xq, xs = ops.quantize_e4m3(x)
    want = ops.gemm(xq, wq, bias=bias, residual=res, act=act, scale_a=xs, scale_w=ws)
    weights = {"w": pack_kblock_swizzled(wq), "w_scale": ws.reshape(())}
    inputs = {"x": x}
    if bias is not None:
        weights["b"] = bias
    if res is not None:
        inputs["res"] = res

    def body(r):
        q, s = r.alloc(padded_token_rows(M) * K), r.alloc(4)
        r.quantize_e4m3(Tensor("x"), q, s, M * K, packed=(M, K))
        r.gemm(q, Weight("w"), Tensor("y"), M, N, K, dtype="e4m3", scale_a=s, scale_w=Weight("w_scale"),
               bias=Weight("b") if bias is not None else None, residual=Tensor("res") if res is not None else None,
               act=act, packed=True, tactic="persistent")
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, weights, inputs, {"y": (BF, (M, N)), "status": (torch.int32, (1,))}, body, repeats=3)
    assert got["status"].item() == 0, hex(got["status"].item())
    assert ops.max_rel_err(got["y"], want) < 1e-2


@pytest.mark.parametrize("case", [(288, 16, 2, 128, "causal", 0), (512, 16, 16, 80, "block", 64)], ids=lambda c: "x".join(map(str, c)))
def test_attention_that_folds_the_amax(tmp_path, case):
    sq, hq, hkv, d, mask, arg = case
    q, k, v = randn(sq, hq * d, seed=121), randn(sq, hkv * d, seed=122), randn(sq, hkv * d, seed=123)

    def body(r):
        o1, o2 = r.alloc(sq * hq * d * 2), r.alloc(sq * hq * d * 2)
        kw = dict(q_rows=sq, kv_rows=sq, q_heads=hq, kv_heads=hkv, head_dim=d, q_stride=hq * d, k_stride=hkv * d,
                  v_stride=hkv * d, o_stride=hq * d, mask=mask, mask_arg=arg)
        amax = r.counter()
        r.attention(Tensor("q"), Tensor("k"), Tensor("v"), o1, algorithm="fa", **kw)
        r.quantize_e4m3(o1, Tensor("q_two_pass"), Tensor("s_two_pass"), sq * hq * d)
        r.attention(Tensor("q"), Tensor("k"), Tensor("v"), o2, amax=amax, **kw)
        r.quantize_e4m3(o2, Tensor("q_folded"), Tensor("s_folded"), sq * hq * d, amax=amax)

    u8, f32 = (torch.uint8, (sq, hq * d)), (torch.float32, (1,))
    got, _ = run_recipe(tmp_path, {}, {"q": q, "k": k, "v": v},
                        {"q_two_pass": u8, "s_two_pass": f32, "q_folded": u8, "s_folded": f32}, body, repeats=2)
    assert torch.equal(got["s_two_pass"], got["s_folded"]) and torch.equal(got["q_two_pass"], got["q_folded"])
    assert got["s_folded"].item() > 0


@pytest.mark.parametrize("shape", [(288, 2048), (50, 1280), (1, 128)], ids=lambda s: "x".join(map(str, s)))
def test_quantize_e4m3_packed_layout_is_bit_exact(tmp_path, shape):
    """Quantisation written in the packed operand layout: same bytes and scale as the oracle, at the addresses
    recipes/layout.py defines (rows past M are padding and not compared)."""
    from aginfer_b200.recipes.layout import padded_token_rows, unpack_kblock_swizzled
    M, K = shape
    x = randn(M, K, seed=131)
    rp = padded_token_rows(M)

    def body(r):
        r.quantize_e4m3(Tensor("x"), Tensor("q"), Tensor("s"), M * K, packed=(M, K))

    got, _ = run_recipe(tmp_path, {}, {"x": x}, {"q": (torch.uint8, (K // 128, rp, 128)), "s": (torch.float32, (1,))},
                        body, repeats=2)
    want_q, want_s = ops.quantize_e4m3(x)
    assert got["s"].view(torch.int32).item() == want_s.reshape(1).view(torch.int32).item()
    unpacked = unpack_kblock_swizzled(got["q"].view(torch.float8_e4m3fn), M)
    assert torch.equal(unpacked.view(torch.uint8), want_q.view(torch.uint8))


SKINNY_CASES = [
    (17, 1536, 1536, "bf16", "bias_gelu_res"), (17, 6144, 1536, "bf16", "bias_gelu"), (17, 1536, 6144, "bf16", "bias_res"),
    (4, 3072, 1536, "bf16", "bias"), (1, 1024, 64, "bf16", "bias"), (16, 1536, 32, "bf16", "bias"),
    (16, 32, 1024, "bf16", "bias"), (50, 1024, 4096, "bf16", "plain"), (64, 4096, 1024, "bf16", "plain"),
    (33, 100, 96, "bf16", "bias"),
    # long K: the bulk-stream tactic cuts these into 4 (or, 4160 = 65 x 64, 2) slices over a thread-block cluster
    (9, 256, 8192, "bf16", "bias_gelu"), (1, 128, 16384, "bf16", "plain"), (25, 520, 4096, "bf16", "bias_res"),
    (17, 1536, 4160, "bf16", "bias_res"),
    (1, 2048, 2048, "e4m3", "plain"), (16, 11008, 2048, "e4m3", "plain"), (64, 2048, 11008, "e4m3", "bias"),
    (64, 2560, 2048, "e4m3", "plain"), (16, 1536, 1536, "e4m3", "plain"), (1, 6144, 1536, "e4m3", "plain"),
]


@pytest.mark.parametrize("tactic", ["skinny", "stream"])
@pytest.mark.parametrize("case", SKINNY_CASES, ids=lambda c: "-".join(map(str, c)))
def test_gemm_skinny(tmp_path, case, tactic):
    M, N, K, dtype, epi = case
    x, wf = randn(M, K, seed=31), randn(N, K, seed=32, std=0.02)
    bias = randn(N, seed=33, std=0.1) if "bias" in epi else None
    res = randn(M, N, seed=34) if "res" in epi else None
    act = "gelu_tanh" if "gelu" in epi else None
    weights, inputs = {}, {"x": x}
    if dtype == "e4m3":
        wq, ws = ops.quantize_e4m3(wf)
        xq, xs = ops.quantize_e4m3(x)
        weights.update({"w": wq, "w_scale": ws.reshape(())})
        want = ops.gemm(xq, wq, bias=bias, residual=res, act=act, scale_a=xs, scale_w=ws)
    else:
        weights["w"] = wf.to(BF)
        want = ops.gemm(x, wf.to(BF), bias=bias, residual=res, act=act)
    if bias is not None:
        weights["b"] = bias
    if res is not None:
        inputs["res"] = res

    def body(r):
        kw = dict(bias=Weight("b") if bias is not None else None, residual=Tensor("res") if res is not None else None,
                  act=act, tactic=tactic)
        if dtype == "e4m3":
            q, s = r.alloc(M * K), r.alloc(4)
            r.quantize_e4m3(Tensor("x"), q, s, M * K)
            r.gemm(q, Weight("w"), Tensor("y"), M, N, K, dtype="e4m3", scale_a=s, scale_w=Weight("w_scale"), **kw)
        else:
            r.gemm(Tensor("x"), Weight("w"), Tensor("y"), M, N, K, **kw)
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, weights, inputs, {"y": (BF, (M, N)), "status": (torch.int32, (1,))}, body, repeats=2)
    assert got["status"].item() == 0, hex(got["status"].item())
    assert ops.max_rel_err(got["y"], want) < 1e-2


@pytest.mark.parametrize("fuse", [True, False], ids=["one_launch", "separate_launches"])
@pytest.mark.parametrize("modulated", [True, False])
def test_fused_layernorm_qkv_linear(tmp_path, fuse, modulated):
    # AdaLN + Q|K|V projections of the action head as one launch, against LN -> three GEMMs in the oracle
    M, K, N = 17, 1536, 1536
    x = (randn(M, K, seed=41).float() * 2 + 0.5).to(BF)
    ws = [randn(N, K, seed=42 + i, std=0.02) for i in range(3)]
    bs = [randn(N, seed=45 + i, std=0.1) for i in range(3)]
    mod = randn(2 * K, seed=48, std=0.3)
    weights = {f"w{i}": ws[i] for i in range(3)} | {f"b{i}": bs[i] for i in range(3)} | {"mod": mod}

    def body(r):
        scratch = r.alloc(M * K * 2)
        ln = {"eps": 1e-5}
        if modulated:
            ln |= {"scale": Weight("mod"), "shift": Weight("mod") + 2 * K}
        out = r.alloc(M * 3 * N * 2)   # column blocks need pointer arithmetic, which caller tensors do not allow
        r.fused_linear(Tensor("x"), [(Weight(f"w{i}"), Weight(f"b{i}"), N) for i in range(3)], out, M, K,
                       ln=ln, ln_scratch=scratch, fuse=fuse, fuse_ln=True)
        from aginfer_b200.recipes import U32
        r.launch("agi_copy_rows_bf16", (296, 1, 1), (256, 1, 1), [out, Tensor("y"), U32(M), U32(3 * N), U32(3 * N), U32(3 * N)])
        r.export_status(Tensor("status"))

    got, stats = run_recipe(tmp_path, weights, {"x": x}, {"y": (BF, (M, 3 * N)), "status": (torch.int32, (1,))}, body,
                            repeats=2)
    assert got["status"].item() == 0
    assert stats["launches_per_enqueue"] == (4 if fuse else 7)
    h = ops.layernorm(x, 1e-5, mod[:K], mod[K:]) if modulated else ops.layernorm(x, 1e-5)
    want = torch.cat([ops.gemm(h, ws[i], bias=bs[i]) for i in range(3)], dim=1)
    assert ops.max_rel_err(got["y"], want) < 1e-2


CLUSTER_CASES = [(17, 1536, 1536, "bias_gelu_res"), (17, 6144, 1536, "bias_gelu"), (17, 1536, 6144, "bias_res"),
                 (17, 4608, 1536, "bias"), (4, 3072, 1536, "bias"), (50, 1024, 4096, "plain"), (1, 2048, 2048, "plain"),
                 (33, 1000, 1024, "bias")]


@pytest.mark.parametrize("case", CLUSTER_CASES, ids=lambda c: "-".join(map(str, c)))
def test_gemm_tcgen05_cluster_split_k(tmp_path, case):
    from aginfer_b200.recipes.builder import tc_cluster_tiling
    M, N, K, epi = case
    assert tc_cluster_tiling(M, N, K, 2) is not None
    x, w = randn(M, K, seed=51), randn(N, K, seed=52, std=0.02)
    bias = randn(N, seed=53, std=0.1) if "bias" in epi else None
    res = randn(M, N, seed=54) if "res" in epi else None
    act = "gelu_tanh" if "gelu" in epi else None
    weights, inputs = {"w": w}, {"x": x}
    if bias is not None:
        weights["b"] = bias
    if res is not None:
        inputs["res"] = res

    def body(r):
        r.gemm(Tensor("x"), Weight("w"), Tensor("y"), M, N, K, bias=Weight("b") if bias is not None else None,
               residual=Tensor("res") if res is not None else None, act=act, tactic="cluster")
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, weights, inputs, {"y": (BF, (M, N)), "status": (torch.int32, (1,))}, body, repeats=3)
    assert got["status"].item() == 0, hex(got["status"].item())
    assert ops.max_rel_err(got["y"], ops.gemm(x, w, bias=bias, residual=res, act=act)) < 1e-2


# (M, widths, K, epilogue, cluster, groups, K blocks per slice); None = the builder's own choice
TCS_CASES = [(17, (1536,), 1536, "bias_gelu_res", None, None, None), (17, (6144,), 1536, "bias_gelu", None, None, None),
             (17, (1536,), 6144, "bias_res", None, None, None), (17, (1536, 1536, 1536), 1536, "bias", None, None, None),
             (17, (1536,), 6144, "bias_res", 1, 12, 8), (17, (6144,), 1536, "bias", 1, 6, 4), (17, (1536,), 512, "plain", 1, 1, 8),
             (16, (1536,), 1536, "bias", 4, 1, 6), (1, (1024,), 512, "bias", 2, 1, 4), (32, (256, 128), 1024, "bias_res", 3, 2, 3),
             (9, (384,), 1152, "plain", 6, 3, 1), (17, (1536,), 6144, "bias_res", 8, 4, 3)]


@pytest.mark.parametrize("case", TCS_CASES, ids=lambda c: "-".join(map(str, c)))
def test_gemm_packed_weight_streaming_tensor_core(tmp_path, case):
    """agi_gemm_tcs_bf16 and its cluster variants: packed bf16 weights, up to 32 tokens, one to three matrices side by
    side, K slices meeting in distributed shared memory, in global slabs, or both."""
    from aginfer_b200.recipes.layout import pack_kblock_swizzled
    M, widths, K, epi, cluster, groups, kb = case
    if kb is not None and cluster * groups * kb < K // 64:
        kb = -(-K // 64 // (cluster * groups))
    x = randn(M, K, seed=61)
    ws = [randn(n, K, seed=62 + i, std=0.02) for i, n in enumerate(widths)]
    bs = [randn(n, seed=70 + i, std=0.1) for i, n in enumerate(widths)] if "bias" in epi else [None] * len(widths)
    total = sum(widths)
    res = randn(M, total, seed=54) if "res" in epi else None
    act = "gelu_tanh" if "gelu" in epi else None
    weights = {f"w{i}": pack_kblock_swizzled(w) for i, w in enumerate(ws)}
    weights.update({f"b{i}": b for i, b in enumerate(bs) if b is not None})
    inputs = {"x": x, **({"res": res} if res is not None else {})}

    def body(r):
        parts = [(Weight(f"w{i}"), Weight(f"b{i}") if bs[i] is not None else None, n) for i, n in enumerate(widths)]
        r.gemm_tcs(Tensor("x"), parts, Tensor("y"), M, K, residual=Tensor("res") if res is not None else None, act=act,
                   cluster=cluster, groups=groups, kb=kb)
        r.export_status(Tensor("status"))

    got, _ = run_recipe(tmp_path, weights, inputs, {"y": (BF, (M, total)), "status": (torch.int32, (1,))}, body, repeats=3)
    assert got["status"].item() == 0, hex(got["status"].item())
    want = torch.cat([ops.gemm(x, w, bias=b) for w, b in zip(ws, bs)], dim=1)
    if act or res is not None:
        want = torch.cat([ops.gemm(x, w, bias=b, residual=None if res is None else res[:, o:o + n], act=act)
                          for w, b, n, o in zip(ws, bs, widths, [sum(widths[:i]) for i in range(len(widths))])], dim=1)
    assert ops.max_rel_err(got["y"], want) < 1e-2
