"""Tiles of the tensor-core GEMM: every shape gets one that the kernel's limits allow, and the way K is summed is a
function of the shape alone."""
import pytest

from aginfer_b200.recipes import RecipeBuilder, Tensor, qwen_vl
from aginfer_b200.recipes.builder import FLAG_GROUPS_FIRST, TC_SCRATCH_BYTES, TK_CLUSTERS, k_runs, tk_grid, tk_tiling
from aginfer_b200.recipes.package import describe

SHAPES = [(16, 128), (130, 256), (2048, 2048), (11008, 2048), (2048, 11008), (3584, 18944), (151, 640)]


@pytest.mark.parametrize("M", [33, 64, 65, 127, 128, 129, 288, 513, 1024, 4097, 8192, 8193, 12000, 20000])
@pytest.mark.parametrize("N,K", SHAPES)
def test_tiles_stay_inside_the_kernels_limits(M, N, K):
    for elem in (1, 2):
        for runs in (None, k_runs(M, N, K, elem)):
            t = tk_tiling(M, (N,), K, elem, runs=runs, clusters=TK_CLUSTERS["agi_gemm_tk_e4m3"] if runs else (1, 2, 4, 8))
            blocks, held = K * elem // 128, -(-t["runs"] // t["C"])
            m_tiles, cols = -(-t["tg"] // 128), -(-t["NB"] // 32) * 32
            assert runs is None or t["runs"] == runs
            assert t["C"] <= t["runs"] and t["runs"] * t["per_run"] >= blocks > (t["runs"] - 1) * t["per_run"]
            assert t["tg"] % 8 == 0 and t["NB"] % 16 == 0 and held * m_tiles * cols <= 512
            assert t["groups"] * t["tg"] >= M and t["tiles"] * t["NB"] >= N and 2 <= t["stages"] <= 8
            ring = t["stages"] * (t["tg"] + t["NB"]) * 128
            last_slot = ring - (t["tg"] + t["NB"]) * 128
            assert 1024 + max(ring, last_slot + m_tiles * 16384) <= t["shared_bytes"] <= 227 * 1024
            assert t["C"] == 1 or t["tiles"] * t["groups"] * t["runs"] * t["NB"] * -(-t["tg"] // 32) * 128 <= TC_SCRATCH_BYTES


@pytest.mark.parametrize("M,N,K,splits,ranks", [(17, 1280, 1280, 8, 4), (128, 1280, 1152, 16, 4), (64, 152064, 2048, 2, 1),
                                                (256, 2048, 2048, 8, 8), (300, 256, 1024, 3, 2), (600, 256, 64, 8, 1)])
def test_tiles_of_256_rows_take_as_many_k_slices_as_can_be_made(M, N, K, splits, ranks):
    r, y = RecipeBuilder({"w": ("BF16", [8])}), Tensor("y")
    r.begin_profile("default", [], [])
    r.gemm(y, y, y, M, N, K, tactic="tcgen05_wide", splits=splits)
    launch = r.profiles[0].launches[-1]
    assert launch["grid"][2] == ranks and launch["kernel"] == "agi_gemm_tk_bf16" + (f"_c{ranks}" if ranks > 1 else "")


@pytest.mark.parametrize("M", [8192, 8193, 8448, 30000])
def test_products_of_many_rows_get_a_launch_from_every_entry_point(M):
    N, K, y = 2048, 1280, Tensor("y")
    r = RecipeBuilder({"w": ("BF16", [8])})
    r.begin_profile("default", [], [])
    before = r.launch_count()
    for dtype in ("bf16", "e4m3"):
        r.gemm(y, y, y, M, N, K, dtype=dtype)
        r.gemm(y, y, y, M, N, K, dtype=dtype, tactic="tcgen05_wide")
        r.gemm_group(y, [(y, None, None, y, N, N), (y, None, None, y, 256, 256)], M, K, dtype=dtype)
        r.gemm_swiglu(y, (y, None, None), (y, None, None), y, M, N, K, dtype=dtype)
    for tactic in ("auto", "persistent", "tcgen05_plan"):
        r.gemm(y, y, y, M, N, K, dtype="e4m3", packed=True, tactic=tactic)
    r.gemm_batch(y, [(y, y)] * 16, y, M, N, K, seg_stride=M * N)
    assert r.launch_count() - before == 12


def test_a_prefill_of_33_images_builds():
    cfg = qwen_vl.VlConfig(images=33, text_tokens=8, v_layers=1, layers=1, vocab=64, v_full_layers=())
    assert cfg.patches == 33 * 256
    for packed in (False, True):
        weights = qwen_vl.synthetic_weights(cfg)
        r = qwen_vl.build_recipe(cfg, describe(qwen_vl.pack_checkpoint(weights) if packed else weights), packed=packed)
        assert r.launch_count() > 20


@pytest.mark.parametrize("wide,text,launches", [(False, 128, 1), (False, 160, 2), (False, 209, 1), (False, 896, 1), (True, 128, 1),
                                                (True, 129, 2), (True, 208, 2), (True, 209, 1), (True, 512, 1)])
def test_gate_and_up_are_two_launches_for_three_token_groups_only(wide, text, launches):
    """Row-major operands; ``text`` + 128 rows of a 3B- or a 7B-shaped layer."""
    kw = dict(hidden=3584, heads=28, kv_heads=4, intermediate=18944) if wide else {}
    cfg = qwen_vl.VlConfig(images=2, text_tokens=text, v_layers=1, layers=1, vocab=64, v_full_layers=(), **kw)
    shapes = {"visual.merger.mlp.0": (5120, 5120), "visual.merger.mlp.2": (cfg.hidden, 5120), **qwen_vl.llm_linears(cfg, 0),
              **{n: s[:2] for n, s in qwen_vl.vision_linears(cfg, 0).items()}}
    weights = {f"{n}.weight": ("F8_E4M3", s) for n, s in shapes.items()} | {f"{n}.weight_scale": ("F32", ()) for n in shapes}
    weights |= {n: ("BF16", (cfg.hidden,)) for n in ("model.layers.0.input_layernorm.weight", "model.norm.weight",
                                                     "model.layers.0.post_attention_layernorm.weight")}
    weights |= {n: ("BF16", (1280,)) for n in ("visual.blocks.0.norm1.weight", "visual.blocks.0.norm2.weight", "visual.merger.ln_q.weight")}
    weights |= {"visual.patch_embed.proj.weight": ("BF16", (1280, cfg.patch_k)), "model.embed_tokens.weight": ("BF16", (64, cfg.hidden))}
    r = qwen_vl.build_recipe(cfg, weights)
    wide_products = [l for l in r.profiles[0].launches if any(a == {"scalar_u32": cfg.intermediate} for a in l["arguments"][13:])
                     and l["kernel"].startswith("agi_gemm_t") and l["arguments"][7] == {"scalar_u32": cfg.hidden}]
    assert len(wide_products) == launches


# (N, K, bytes an element, packed): the row counts from which on K is cut into another number of runs, up to 1600 rows.
# Recorded when FP8 stacks were first held to it; a change here changes the output bits of packaged models.
K_RUNS = {
    (1280, 1280, 1, False): "1:4 65:5 128:1",
    (3840, 1280, 1, False): "1:4 65:5 128:1",
    (1280, 3456, 1, False): "1:1 65:9 128:4 193:3 321:2 561:1",
    (5120, 5120, 1, False): "1:2 65:4 128:3 129:1 145:3 161:1",
    (2048, 5120, 1, False): "1:8 65:10 128:4 129:3 145:4 161:3 241:2 257:3 289:2 321:3 337:2 449:3 481:1",
    (3584, 5120, 1, False): "1:4 65:6 128:2 225:1",
    (2048, 2048, 1, False): "1:8 128:4 129:3 193:1",
    (11008, 2048, 1, False): "1:1 65:2 128:1",
    (2048, 11008, 1, False): "1:8 65:10 128:4 129:3 145:4 161:3 1249:2 1297:3 1345:2",
    (3584, 3584, 1, False): "1:4 65:6 128:2 193:1",
    (18944, 3584, 1, False): "1:1",
    (3584, 18944, 1, False): "1:4 65:6 128:4 321:3 337:4 353:3 769:2 1171:1",
    (1280, 1216, 2, False): "1:1 65:7 128:4 193:3 257:2 449:1",
    (2048, 11008, 1, True): "1:8 65:4 129:3 145:4 161:3 768:1",
    (3584, 18944, 1, True): "1:4 321:3 337:4 353:3 768:1",
}


@pytest.mark.parametrize("shape", K_RUNS, ids=lambda s: "x".join(map(str, s)))
def test_the_order_of_the_sum_over_k_is_the_recorded_one(shape):
    N, K, elem, packed = shape
    found, last = [], None
    for M in range(1, 1601):
        runs = k_runs(M, N, K, elem, packed)
        if runs != last:
            found.append(f"{M}:{runs}")
        last = runs
    assert " ".join(found) == K_RUNS[shape]


@pytest.mark.parametrize("tiles,groups,grid", [(96, 1, (96, 1)), (96, 3, (3, 96)), (1, 4, (4, 1)), (65535, 2, (2, 65535)),
                                               (65536, 2, (65536, 2)), (70000, 1, (70000, 1)), (1, 65535, (65535, 1)),
                                               (1, 65536, (1, 65536)), (16, 65792, (16, 65792)), (65535, 89241, (65535, 89241)),
                                               (70000, 70000, (70000, 70000))])
def test_token_groups_run_side_by_side_where_the_grid_takes_the_tiles(tiles, groups, grid):
    assert tk_grid({"tiles": tiles, "groups": groups}) == grid


def test_more_token_groups_than_a_grid_takes_stay_where_the_launch_refuses_them():
    M, N, K, y = 33554432, 64, 64, Tensor("y")
    r = RecipeBuilder({"w": ("BF16", [8])})
    r.begin_profile("default", [], [])
    before = r.launch_count()
    r.gemm(y, y, y, M, N, K)
    r.gemm_group(y, [(y, None, None, y, N, N)] * 2, M, K)
    r.gemm_batch(y, [(y, y)] * 2, y, M, N, K, seg_stride=M * N)
    launches = r.profiles[0].launches[before:]
    assert len(launches) == 3 and all(l["grid"][0] <= 4 and l["grid"][1] > 65535 for l in launches)


def order(M, N, K, emit):
    """(grid, groups first) of the launch that ``emit`` adds for token rows M."""
    y, r = Tensor("y"), RecipeBuilder({"w": ("BF16", [8])})
    r.begin_profile("default", [], [])
    emit(r, y, M, N, K)
    launch = r.profiles[0].launches[-1]
    flags = launch["arguments"][{"agi_gemm_tcq_e4m3": 13, "agi_gemm_tc_bf16_x16": 8}.get(launch["kernel"], 9)]["scalar_u32"]
    return launch["grid"], bool(flags & FLAG_GROUPS_FIRST)


EMIT = {"gemm": lambda r, y, M, N, K: r.gemm(y, y, y, M, N, K),
        "group": lambda r, y, M, N, K: r.gemm_group(y, [(y, None, None, y, N // 2, N // 2)] * 2, M, K),
        "swiglu": lambda r, y, M, N, K: r.gemm_swiglu(y, (y, None, None), (y, None, None), y, M, N // 2, K),
        "batch": lambda r, y, M, N, K: r.gemm_batch(y, [(y, y)] * 2, y, M, N // 2, K, seg_stride=M * N),
        "persistent": lambda r, y, M, N, K: r.gemm(y, y, y, M, N, 2 * K, dtype="e4m3", packed=True, tactic="persistent")}


@pytest.mark.parametrize("kind", EMIT)
@pytest.mark.parametrize("M,N,K,first", [(288, 22016, 2048, True), (4096, 2048, 2048, True), (16384, 2048, 1280, True),
                                         (16384, 2048, 2048, False), (16384, 11008, 2048, False), (16384, 22016, 2048, True),
                                         (8192, 2048, 3072, True), (8192, 2048, 3840, False)])
def test_token_groups_run_side_by_side_unless_the_tokens_are_the_larger_operand_and_pass_l2(kind, M, N, K, first):
    grid, flag = order(M, N, K, EMIT[kind])
    assert flag == (first and not (kind == "persistent" and M * 2 * K > 48 << 20))
    if kind != "persistent":
        t = tk_tiling(M, (N,) if kind == "gemm" else (N // 2,) if kind == "swiglu" else (N // 2,) * 2, K, 2, swiglu=kind == "swiglu",
                      clusters=(1, 2, 4, 8) if kind == "gemm" else (1,))
        assert grid == [*((t["groups"], t["tiles"]) if first else (t["tiles"], t["groups"])), t["C"]]
