"""What the speed of this framework is measured on: packaged recipes replayed through ``aginfer_b200.runner.Runner``.

Each case is one package (weights and a launch recipe, as ``modelc`` writes them) that a serving process has loaded,
and one pass is one ``Runner.run``: a request's tensors in, the recipe's outputs in the caller's buffers.  A process
keeps its package loaded from request to request, so the package follows from the case alone and is kept here, while
inputs (and the output buffers that receive the answer) are new for every seed.  Packages run with programmatic
dependent launch, as ``bench.py`` runs them.

Families, all at the widths of the repository's own configurations:

* ``linear``   FP8 linears on one activation matrix: dynamic per-tensor quantisation, then the scaled GEMM (row-major
               weights or the packed layout).  The (N, K) grid of the GEMM sweep, one token to a long prefill.
* ``layer``    one decoder layer over a whole prompt, BF16 or FP8 weights.
* ``chunk``    the flow-matching action head: an action chunk of some Euler steps (batch 1, few tokens, weights
               streamed once a step).
* ``prefill``  vision tower, merger and decoder layers in FP8 from pixels and token ids to hidden states and K/V cache.
* ``episode``  prefill of the wider backbone followed by the BF16 action expert's Euler steps over its K/V cache.

Widths, token counts and step counts are the real ones; the block stacks of ``prefill`` and ``episode`` are cut to a
few blocks each (every block of a stack is the same launches): per-tensor FP8 quantisation amplifies a last-bit
difference from block to block, so only the output of a short stack says whether the arithmetic is the same.
"""
from __future__ import annotations

import math
import tempfile
from collections import OrderedDict
from pathlib import Path

import torch

from aginfer_b200 import runtime as rt
from aginfer_b200.build import CUBIN, build_kernels
from aginfer_b200.container import AimWriter, VariantPayload
from aginfer_b200.planfmt import compile_execution_plan
from aginfer_b200.recipes import RecipeBuilder, Tensor, Weight, decoder_layer, dit, io, lingbot, qwen_vl
from aginfer_b200.recipes.layout import pack_kblock_swizzled, padded_token_rows
from aginfer_b200.recipes.package import TOOLCHAIN
from aginfer_b200.runner import Runner
from aginfer_b200.target import CudaArch, Platform

# (N, K) of the repository's FP8 GEMM sweep
SWEEP = ((2048, 2048), (11008, 2048), (2048, 11008), (2560, 2048), (1536, 1536), (6144, 1536))
VOCAB = 8192          # rows of the embedding table: a gather reads one row a token, whatever the table's length
L2_BYTES = 126 << 20
MAX_LOADED = 20       # packages kept loaded (a few GB all together)


def listed() -> list[dict]:
    return [
        # the smallest call: one projection of one token
        {"name": "linear_1tok", "family": "linear", "tokens": 1, "n": 2048, "k": 2048, "sweep": False, "packed": False},
        # the whole (N, K) grid for a handful of tokens: weight streaming
        {"name": "sweep_16tok", "family": "linear", "tokens": 16, "n": 0, "k": 0, "sweep": True, "packed": False},
        # the same for a short prompt, and for a long one in the packed layout
        {"name": "sweep_288tok", "family": "linear", "tokens": 288, "n": 0, "k": 0, "sweep": True, "packed": False},
        {"name": "sweep_1024tok_packed", "family": "linear", "tokens": 1024, "n": 0, "k": 0, "sweep": True, "packed": True},
        # one BF16 decoder layer over the 288-token prompt, one FP8 layer over an odd, short one
        {"name": "layer_bf16_288", "family": "layer", "tokens": 288, "width": 2048, "fp8": False},
        {"name": "layer_fp8_77", "family": "layer", "tokens": 77, "width": 2048, "fp8": True},
        # the action head as it is deployed: 16 blocks, 4 steps, 16 actions, 300 context tokens
        {"name": "chunk_16x4", "family": "chunk", "layers": 16, "steps": 4, "context": 300, "horizon": 16},
        # a single-step chunk of a shallow head with a short, odd context; a long horizon (more than 32 tokens)
        {"name": "chunk_4x1_short", "family": "chunk", "layers": 4, "steps": 1, "context": 77, "horizon": 8},
        {"name": "chunk_4x2_long", "family": "chunk", "layers": 4, "steps": 2, "context": 288, "horizon": 49},
        # backbone prefill: packed weights with the 288-token prefix, row-major ones with one image and an odd prompt
        {"name": "prefill_288_packed", "family": "prefill", "images": 2, "text": 160, "v_layers": 4, "layers": 4, "packed": True},
        {"name": "prefill_101", "family": "prefill", "images": 1, "text": 37, "v_layers": 4, "layers": 4, "packed": False},
        # an episode: three cameras, 64 text tokens, ten steps of the action expert
        {"name": "episode", "family": "episode", "images": 3, "text": 64, "v_layers": 4, "layers": 4, "e_layers": 5,
         "steps": 10, "horizon": 50, "packed": True},
    ]


def _log(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    family = rng.choice(("linear", "linear", "layer", "layer", "chunk", "chunk", "prefill", "prefill", "episode"))
    if family == "linear":
        tokens, sweep = _log(rng, 1, 1024), rng.random() < 0.5
        return {"family": family, "tokens": tokens, "n": 0 if sweep else 128 * _log(rng, 12, 86),
                "k": 0 if sweep else 128 * _log(rng, 12, 86), "sweep": sweep, "packed": tokens > 64 and rng.random() < 0.5}
    if family == "layer":
        return {"family": family, "tokens": _log(rng, 16, 768), "width": rng.choice((2048, 2048, 3584)),
                "fp8": rng.random() < 0.5}
    if family == "chunk":
        return {"family": family, "layers": 2 * rng.randint(2, 8), "steps": rng.randint(1, 4), "context": _log(rng, 64, 600),
                "horizon": _log(rng, 8, 63)}
    if family == "prefill":
        return {"family": family, "images": rng.randint(1, 3), "text": _log(rng, 8, 256), "v_layers": rng.randint(2, 4),
                "layers": rng.randint(2, 4), "packed": rng.random() < 0.5}
    return {"family": family, "images": rng.randint(1, 3), "text": _log(rng, 8, 128), "v_layers": 2, "layers": rng.randint(2, 3),
            "e_layers": rng.randint(4, 6), "steps": rng.randint(2, 10), "horizon": _log(rng, 8, 63), "packed": rng.random() < 0.5}


# ---- what a case stands for -----------------------------------------------------------------------------

def _shapes(case: dict) -> list[tuple[int, int]]:
    return list(SWEEP) if case["sweep"] else [(case["n"], case["k"])]


def _layer_config(case: dict) -> decoder_layer.LayerConfig:
    wide = {} if case["width"] == 2048 else dict(hidden=3584, heads=28, kv_heads=4, intermediate=18944)
    return decoder_layer.LayerConfig(tokens=case["tokens"], fp8=case["fp8"], **wide)


def _chunk_config(case: dict) -> dit.DitConfig:
    return dit.DitConfig(layers=case["layers"], steps=case["steps"], backbone_tokens=case["context"], horizon=case["horizon"])


def _backbone(case: dict, base: qwen_vl.VlConfig) -> qwen_vl.VlConfig:
    from dataclasses import replace
    return replace(base, images=case["images"], text_tokens=case["text"], v_layers=case["v_layers"],
                   v_full_layers=(case["v_layers"] - 1,), layers=case["layers"], vocab=VOCAB)


def _episode_config(case: dict) -> lingbot.EpisodeConfig:
    return lingbot.EpisodeConfig(backbone=_backbone(case, lingbot.BACKBONE_7B), e_layers=case["e_layers"],
                                 steps=case["steps"], horizon=case["horizon"])


# ---- packages -------------------------------------------------------------------------------------------

def _weights(case: dict) -> dict:
    """A random-init checkpoint of the case's architecture, made on the GPU: linears ~ N(0, 0.02) (E4M3 ones
    quantised per tensor by amax / 448), biases ~ N(0, 0.02), norm gains one; padding rows and columns zero."""
    g = torch.Generator(device="cuda").manual_seed(20)
    out: dict[str, torch.Tensor] = {}

    def dense(name: str, shape, live=None) -> None:
        w = torch.zeros(shape, device="cuda")
        box = tuple(slice(0, n) for n in (live or shape))
        w[box] = torch.randn([s.stop for s in box], generator=g, device="cuda") * 0.02
        out[name] = w.to(torch.bfloat16)

    def fp8(name: str, n: int, k: int, n_live: int | None = None, k_live: int | None = None) -> None:
        w = torch.zeros(n, k, device="cuda")
        w[:n_live or n, :k_live or k] = torch.randn(n_live or n, k_live or k, generator=g, device="cuda") * 0.02
        scale = w.abs().max() / 448.0
        out[f"{name}.weight"] = (w / scale).clamp(-448, 448).to(torch.float8_e4m3fn)
        out[f"{name}.weight_scale"] = scale.reshape(())

    def ones(name: str, n: int) -> None:
        out[name] = torch.ones(n, dtype=torch.bfloat16, device="cuda")

    def backbone(cfg: qwen_vl.VlConfig) -> None:
        dense("visual.patch_embed.proj.weight", (cfg.v_hidden, cfg.patch_k), (cfg.v_hidden, cfg.patch_elems))
        for i in range(cfg.v_layers):
            for name, (n, k, n_live, k_live) in qwen_vl.vision_linears(cfg, i).items():
                fp8(name, n, k, n_live, k_live)
                dense(f"{name}.bias", (n,), (n_live,))
            ones(f"visual.blocks.{i}.norm1.weight", cfg.v_hidden)
            ones(f"visual.blocks.{i}.norm2.weight", cfg.v_hidden)
        ones("visual.merger.ln_q.weight", cfg.v_hidden)
        for name, n in (("visual.merger.mlp.0", cfg.merged_dim), ("visual.merger.mlp.2", cfg.hidden)):
            fp8(name, n, cfg.merged_dim)
            dense(f"{name}.bias", (n,))
        dense("model.embed_tokens.weight", (cfg.vocab, cfg.hidden))
        for i in range(cfg.layers):
            for name, (n, k) in qwen_vl.llm_linears(cfg, i).items():
                fp8(name, n, k)
                if name.endswith(("q_proj", "k_proj", "v_proj")):
                    dense(f"{name}.bias", (n,))
            ones(f"model.layers.{i}.input_layernorm.weight", cfg.hidden)
            ones(f"model.layers.{i}.post_attention_layernorm.weight", cfg.hidden)
        ones("model.norm.weight", cfg.hidden)

    if case["family"] == "linear":
        for i, (n, k) in enumerate(_shapes(case)):
            fp8(f"linear{i}", n, k)
    elif case["family"] == "layer":
        cfg, prefix = _layer_config(case), decoder_layer.L
        for name, (n, k) in decoder_layer.linear_shapes(cfg).items():
            if cfg.fp8:
                fp8(f"{prefix}.{name}", n, k)
            else:
                dense(f"{prefix}.{name}.weight", (n, k))
            if name.endswith(("q_proj", "k_proj", "v_proj")):
                dense(f"{prefix}.{name}.bias", (n,))
        ones(f"{prefix}.input_layernorm.weight", cfg.hidden)
        ones(f"{prefix}.post_attention_layernorm.weight", cfg.hidden)
    elif case["family"] == "chunk":
        for name, shape in sorted(dit.weight_shapes(_chunk_config(case)).items()):
            dense(name, shape)
    elif case["family"] == "prefill":
        backbone(_backbone(case, qwen_vl.VlConfig()))
    else:
        cfg = _episode_config(case)
        backbone(cfg.backbone)
        for name, shape in lingbot.expert_shapes(cfg).items():
            if name.endswith(("norm.weight", "layernorm.weight")):
                ones(name, shape[0])
            elif name.endswith(("action_in.weight", "state_in.weight")):
                dense(name, shape, (shape[0], cfg.action_dim))
            elif name.rsplit(".", 1)[0].endswith("action_out"):
                dense(name, shape, (cfg.action_dim, *shape[1:]))
            else:
                dense(name, shape)
    if case.get("packed"):
        out = {k: pack_kblock_swizzled(v.cpu()) if v.dtype == torch.float8_e4m3fn and v.dim() == 2 else v
               for k, v in out.items()}
    return out


def _linear_recipe(case: dict, weights) -> RecipeBuilder:
    """Every activation width is quantised once and multiplied with each matrix of that width."""
    M, shapes, packed = case["tokens"], _shapes(case), case["packed"]
    r = RecipeBuilder(weights)
    r.begin_profile("default", [io(f"x{k}", "BF16", [M, k]) for k in sorted({k for _, k in shapes})],
                    [*(io(f"y{i}", "BF16", [M, n]) for i, (n, _) in enumerate(shapes)), io("status", "I32", [1])])
    for k in sorted({k for _, k in shapes}):
        q, scale = r.alloc((padded_token_rows(M) if packed else M) * k), r.alloc(4)
        r.quantize_e4m3(Tensor(f"x{k}"), q, scale, M * k, packed=(M, k) if packed else None)
        for i, (n, depth) in enumerate(shapes):
            if depth == k:
                r.gemm(q, Weight(f"linear{i}.weight"), Tensor(f"y{i}"), M, n, k, dtype="e4m3", scale_a=scale,
                       scale_w=Weight(f"linear{i}.weight_scale"), packed=packed)
    r.export_status(Tensor("status"))
    return r


def _recipe(case: dict, weights) -> RecipeBuilder:
    if case["family"] == "linear":
        return _linear_recipe(case, weights)
    if case["family"] == "layer":
        return decoder_layer.build_recipe(_layer_config(case), weights)
    if case["family"] == "chunk":
        return dit.build_recipe(_chunk_config(case), weights)
    if case["family"] == "prefill":
        return qwen_vl.build_recipe(_backbone(case, qwen_vl.VlConfig()), weights, packed=case["packed"])
    return lingbot.build_recipe(_episode_config(case), weights, packed=case["packed"])


def _package(case: dict, path: Path) -> None:
    """The case's ``.aim``: what ``modelc compile`` writes, without the checkpoint directory in between."""
    names = {torch.float32: "F32", torch.bfloat16: "BF16", torch.float8_e4m3fn: "F8_E4M3"}
    weights = _weights(case)
    recipe = _recipe(case, {k: (names[v.dtype], tuple(v.shape)) for k, v in weights.items()})
    blob = torch.zeros(recipe.weight_bytes, dtype=torch.uint8, device="cuda")
    for name, t in weights.items():
        raw = t.contiguous().reshape(-1).view(torch.uint8)
        blob[recipe.weight_offsets[name]:recipe.weight_offsets[name] + raw.numel()] = raw.to("cuda")
    payload = blob.cpu().numpy().data
    plan = compile_execution_plan(recipe.plan(), CudaArch.SM100, weight_size=recipe.weight_bytes)
    cubin = (CUBIN if CUBIN.exists() else build_kernels()).read_bytes()
    AimWriter.write(path, platform=Platform.LINUX_X86_64_GNU, manifest={"toolchain": TOOLCHAIN, "profiles": []}, graph={},
                    tensors={"alignment": 256, "count": 0, "items": []}, verify=False,
                    variants=[VariantPayload(CudaArch.SM100, cubin, payload, plan.data)])


_loaded: "OrderedDict[tuple, Runner]" = OrderedDict()


def _runner(case: dict) -> Runner:
    """The loaded package of a case, as a serving process keeps it (the file is gone once it is mapped)."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _loaded:
        while len(_loaded) >= MAX_LOADED:
            _loaded.popitem(last=False)
        with tempfile.TemporaryDirectory(prefix="agi_perf_") as tmp:
            _package(case, Path(tmp) / "model.aim")
            torch.cuda.empty_cache()
            _loaded[key] = Runner(Path(tmp) / "model.aim", flags=rt.PROGRAMMATIC_LAUNCH)
    _loaded.move_to_end(key)
    return _loaded[key]


# ---- a request ------------------------------------------------------------------------------------------

def prepare(case: dict, seed: int) -> dict:
    runner = _runner(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    # hidden states, backbone features, robot state and noise ~ N(0, 1); pixels ~ U(0, 1); random token ids
    inputs = {}
    for t in runner.inputs:
        if t.name == "pixels":
            inputs[t.name] = torch.rand(t.shape, generator=g, device="cuda")
        elif t.name == "input_ids":
            inputs[t.name] = torch.randint(0, VOCAB, t.shape, generator=g, device="cuda", dtype=torch.int32)
        elif t.name == "positions":
            cfg = _backbone(case, qwen_vl.VlConfig()) if case["family"] == "prefill" else _episode_config(case).backbone
            inputs[t.name] = qwen_vl.rope_positions(cfg).cuda()
        else:
            inputs[t.name] = torch.randn(t.shape, generator=g, device="cuda").to(torch.bfloat16)
    return {"runner": runner, "inputs": inputs, "outputs": runner.empty_outputs()}


def run(state: dict) -> dict:
    return state["runner"].run(state["inputs"], state["outputs"])


def work(case: dict) -> dict:
    """Bytes: weights, inputs and outputs, each once; weights of a denoising loop once a step where the loop's
    weights are more than the L2 cache holds, once otherwise.  Flops: the matrix products (attention left out)."""
    if case["family"] == "linear":
        M, shapes = case["tokens"], _shapes(case)
        return {"bytes": sum(n * k + 2 * M * n for n, k in shapes) + sum(2 * M * k for k in {k for _, k in shapes}),
                "flops": sum(2 * M * n * k for n, k in shapes)}
    if case["family"] == "layer":
        a = decoder_layer.algorithmic(_layer_config(case))
        return {"bytes": a["weight_bytes"] + 4 * case["tokens"] * case["width"], "flops": a["flops"]}
    if case["family"] == "chunk":
        cfg = _chunk_config(case)
        a = dit.algorithmic_bytes(cfg)
        loops = cfg.steps if a["per_step"] > L2_BYTES else 1
        return {"bytes": a["once"] + loops * a["per_step"] + 2 * cfg.backbone_tokens * cfg.backbone_dim,
                "flops": cfg.steps * cfg.tokens * a["per_step"]
                + 2 * cfg.backbone_tokens * cfg.backbone_dim * cfg.hidden * 2 * ((cfg.layers + 1) // 2)}
    bb = _backbone(case, qwen_vl.VlConfig()) if case["family"] == "prefill" else _episode_config(case).backbone
    a = qwen_vl.algorithmic(bb)
    total = (a["fp8_weight_bytes"] + a["bf16_weight_bytes"] + 4 * bb.images * bb.channels * bb.image_size ** 2
             + 2 * bb.tokens * (bb.hidden + 2 * bb.layers * bb.kv_dim))
    if case["family"] == "prefill":
        return {"bytes": total, "flops": a["flops"]}
    e = lingbot.algorithmic(_episode_config(case))
    loops = case["steps"] if 2 * e["expert_params"] > L2_BYTES else 1
    return {"bytes": total + 2 * e["expert_params"] * loops, "flops": a["flops"] + e["expert_flops"]}


def tolerance(case: dict) -> dict:
    """Quantisation is bit-exact and accumulation fp32, so a single product differs by its bf16 rounding only.  A block
    stack in FP8 moves by more: one rounding upstream of a per-tensor amax moves the codes of a whole operand."""
    if case["family"] == "linear" or (case["family"] == "layer" and not case["fp8"]):
        return {"rel": 1e-2}
    return {"rel": 2e-2}
