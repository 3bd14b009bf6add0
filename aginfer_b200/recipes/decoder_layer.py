"""Launch recipe of one Qwen2.5-VL-style decoder layer (prefill): RMSNorm -> QKV (+bias) -> 1-D RoPE ->
GQA causal attention -> O projection + residual -> RMSNorm -> gate/up -> SwiGLU -> down + residual.

Default shape: hidden 2048, 16 query / 2 KV heads of 128, SwiGLU 11008, eps 1e-6, theta 1e6, 288 tokens,
BF16 weights.  ``fp8=True`` builds the same layer with E4M3 linear weights and per-tensor fp32 scales
(``<name>.weight_scale``, ModelOpt style); activations are then quantised per tensor before every GEMM.
Checkpoint names follow Hugging Face (``model.layers.0.self_attn.q_proj.weight`` ...), so q/k/v are not
adjacent in the packed blob; above 32 tokens Q | K | V are one grouped launch writing column blocks of one buffer and
SwiGLU runs in the epilogue of gate | up (fewer tokens and other GEMM tactics: one launch per projection).
"""
from __future__ import annotations

from dataclasses import dataclass

from .builder import RecipeBuilder, Tensor, Weight, io


@dataclass(frozen=True)
class LayerConfig:
    hidden: int = 2048
    heads: int = 16
    kv_heads: int = 2
    head_dim: int = 128
    intermediate: int = 11008
    tokens: int = 288
    eps: float = 1e-6
    theta: float = 1e6
    fp8: bool = False

    @property
    def q_dim(self) -> int:
        return self.heads * self.head_dim

    @property
    def kv_dim(self) -> int:
        return self.kv_heads * self.head_dim


L = "model.layers.0"
LINEARS = ("self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj", "mlp.gate_proj",
           "mlp.up_proj", "mlp.down_proj")


def linear_shapes(cfg: LayerConfig) -> dict[str, tuple[int, int]]:
    H, I = cfg.hidden, cfg.intermediate
    return {"self_attn.q_proj": (cfg.q_dim, H), "self_attn.k_proj": (cfg.kv_dim, H), "self_attn.v_proj": (cfg.kv_dim, H),
            "self_attn.o_proj": (H, cfg.q_dim), "mlp.gate_proj": (I, H), "mlp.up_proj": (I, H), "mlp.down_proj": (H, I)}


def synthetic_weights(cfg: LayerConfig, seed: int = 0, std: float = 0.02) -> dict:
    """BF16 ~ N(0, std) linears, RMSNorm gains 1.0, small QKV biases; with ``cfg.fp8`` the linears are
    quantised per tensor by amax / 448 to E4M3 and their fp32 scales stored beside them."""
    import torch
    g = torch.Generator().manual_seed(seed)
    out = {}
    for name, shape in linear_shapes(cfg).items():
        w = torch.randn(shape, generator=g) * std
        if cfg.fp8:
            scale = w.abs().max() / 448.0
            out[f"{L}.{name}.weight"] = (w / scale).clamp(-448, 448).to(torch.float8_e4m3fn)
            out[f"{L}.{name}.weight_scale"] = scale.reshape(()).float()
        else:
            out[f"{L}.{name}.weight"] = w.to(torch.bfloat16)
    for name in ("q_proj", "k_proj", "v_proj"):
        out[f"{L}.self_attn.{name}.bias"] = (torch.randn(linear_shapes(cfg)[f"self_attn.{name}"][0], generator=g) * std
                                             ).to(torch.bfloat16)
    out[f"{L}.input_layernorm.weight"] = torch.ones(cfg.hidden, dtype=torch.bfloat16)
    out[f"{L}.post_attention_layernorm.weight"] = torch.ones(cfg.hidden, dtype=torch.bfloat16)
    return out


def synthetic_input(cfg: LayerConfig, seed: int = 0):
    import torch
    g = torch.Generator().manual_seed(seed + 1000)
    return torch.randn(cfg.tokens, cfg.hidden, generator=g).to(torch.bfloat16)


def build_recipe(cfg: LayerConfig, weights, gemm_tactic: str = "auto") -> RecipeBuilder:
    """``weights``: name -> (dtype, shape) as from ``package.describe``."""
    S, H, I, D = cfg.tokens, cfg.hidden, cfg.intermediate, cfg.head_dim
    qkv_dim = cfg.q_dim + 2 * cfg.kv_dim
    r = RecipeBuilder(weights)
    r.begin_profile("default", [io("hidden_in", "BF16", [S, H])], [io("hidden_out", "BF16", [S, H])])
    BF = 2
    normed, qkv, attn = r.alloc(S * H * BF), r.alloc(S * qkv_dim * BF), r.alloc(S * cfg.q_dim * BF)
    resid, gate_up, act = r.alloc(S * H * BF), r.alloc(S * 2 * I * BF), r.alloc(S * I * BF)
    quant, scale = r.alloc(S * max(H, I, cfg.q_dim)), r.alloc(4)

    grouped = gemm_tactic == "auto" and H % 128 == 0     # projections that share their input share a launch

    def quantize(x, K, amax=None):
        """FP8 layers quantise each GEMM input once per tensor (amax / 448) into ``quant``."""
        if cfg.fp8:
            r.quantize_e4m3(x, quant, scale, S * K, amax=amax)

    def linear(x, name, y, N, K, **kw):
        """One projection (FP8: of the input last quantised)."""
        w = Weight(f"{L}.{name}.weight")
        if cfg.fp8:
            r.gemm(quant, w, y, S, N, K, dtype="e4m3", scale_a=scale, scale_w=Weight(f"{L}.{name}.weight_scale"),
                   tactic=gemm_tactic, **kw)
        else:
            r.gemm(x, w, y, S, N, K, tactic=gemm_tactic, **kw)

    def norm(x, name):
        """RMSNorm into ``normed``, quantised for an FP8 layer (the norm then leaves max |y| behind)."""
        amax = r.counter() if cfg.fp8 else None
        r.rmsnorm(x, Weight(f"{L}.{name}.weight"), normed, S, H, cfg.eps, amax=amax)
        quantize(normed, H, amax)

    weight_scale = lambda name: Weight(f"{L}.{name}.weight_scale") if cfg.fp8 else None
    operand, dtype, scale_a = (quant, "e4m3", scale) if cfg.fp8 else (normed, "bf16", None)
    norm(Tensor("hidden_in"), "input_layernorm")
    projections, col = [], 0
    for name, width in (("self_attn.q_proj", cfg.q_dim), ("self_attn.k_proj", cfg.kv_dim), ("self_attn.v_proj", cfg.kv_dim)):
        projections.append((name, qkv + col * BF, width))
        col += width
    if grouped and S > 32:       # up to 32 tokens: the weight-streaming kernel, one launch each
        r.gemm_group(operand, [(Weight(f"{L}.{name}.weight"), Weight(f"{L}.{name}.bias"), weight_scale(name), y, width, qkv_dim)
                               for name, y, width in projections], S, H, dtype=dtype, scale_a=scale_a, split=True)
    else:
        for name, y, width in projections:
            linear(normed, name, y, width, H, bias=Weight(f"{L}.{name}.bias"), ldy=qkv_dim)
    r.rope(qkv, S, cfg.heads + cfg.kv_heads, D, qkv_dim, cfg.theta)
    # the streaming kernel (more than 64 query rows) can leave max |o| behind
    attn_amax = r.counter() if cfg.fp8 and S > 64 and D in (80, 128) else None
    r.attention(qkv, qkv + cfg.q_dim * BF, qkv + (cfg.q_dim + cfg.kv_dim) * BF, attn, q_rows=S, kv_rows=S,
                q_heads=cfg.heads, kv_heads=cfg.kv_heads, head_dim=D, q_stride=qkv_dim, k_stride=qkv_dim,
                v_stride=qkv_dim, o_stride=cfg.q_dim, mask="causal", amax=attn_amax)
    quantize(attn, cfg.q_dim, attn_amax)
    linear(attn, "self_attn.o_proj", resid, H, cfg.q_dim, residual=Tensor("hidden_in"))
    norm(resid, "post_attention_layernorm")
    act_amax = r.counter() if cfg.fp8 else None
    if grouped and S > 32:
        part = lambda name: (Weight(f"{L}.{name}.weight"), None, weight_scale(name))
        r.gemm_swiglu(operand, part("mlp.gate_proj"), part("mlp.up_proj"), act, S, I, H, dtype=dtype, scale_a=scale_a, amax=act_amax)
    else:
        linear(normed, "mlp.gate_proj", gate_up, I, H, ldy=2 * I)
        linear(normed, "mlp.up_proj", gate_up + I * BF, I, H, ldy=2 * I)
        r.swiglu(gate_up, gate_up + I * BF, act, S, I, 2 * I, amax=act_amax)
    quantize(act, I, act_amax)
    linear(act, "mlp.down_proj", Tensor("hidden_out"), H, I, residual=resid)
    return r


def algorithmic(cfg: LayerConfig) -> dict[str, int]:
    """Weight bytes and flops of the layer (what the roofline floors are computed from)."""
    params = sum(n * k for n, k in linear_shapes(cfg).values())
    return {"weight_bytes": params * (1 if cfg.fp8 else 2), "flops": 2 * cfg.tokens * params, "params": params}
