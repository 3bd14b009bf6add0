"""Streaming attention at the edges of its row groups (16), row blocks (32), key tiles (64) and key chunks (4 tiles)."""
from __future__ import annotations

import pytest
import torch

from aginfer_b200.recipes import Tensor
from oracle import ops
from tests.gpu_util import MAX_REL, run_recipe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("case", [
    (1, 1, 2, 1, 128, "none", 0), (16, 63, 2, 2, 80, "none", 0), (17, 64, 3, 1, 48, "none", 0), (32, 65, 2, 1, 64, "none", 0),
    (33, 256, 2, 2, 128, "none", 0), (65, 257, 2, 1, 80, "none", 0), (257, 257, 2, 1, 128, "causal", 0),
    (49, 561, 2, 1, 128, "causal", 512), (320, 320, 2, 2, 80, "block", 320), (130, 130, 2, 2, 80, "block", 65),
], ids=lambda c: "x".join(map(str, c)))
def test_attention_at_chunk_edges(tmp_path, case):
    sq, skv, hq, hkv, d, mask, arg = case
    g = torch.Generator().manual_seed(3)
    q, k, v = (torch.randn(n, h * d, generator=g).to(BF) for n, h in ((sq, hq), (skv, hkv), (skv, hkv)))
    got, _ = run_recipe(tmp_path, {}, {"q": q, "k": k, "v": v}, {"o": (BF, (sq, hq * d))}, lambda r: r.attention(
        Tensor("q"), Tensor("k"), Tensor("v"), Tensor("o"), q_rows=sq, kv_rows=skv, q_heads=hq, kv_heads=hkv,
        head_dim=d, q_stride=hq * d, k_stride=hkv * d, v_stride=hkv * d, o_stride=hq * d, mask=mask, mask_arg=arg,
        algorithm="fa"))
    want = ops.attention(q.view(sq, hq, d), k.view(skv, hkv, d), v.view(skv, hkv, d), mask=mask, mask_arg=arg)
    assert ops.max_rel_err(got["o"], want.reshape(sq, -1)) < MAX_REL
