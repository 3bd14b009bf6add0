"""Tiles of the tensor-core GEMM: every shape gets one that the kernel's limits allow, and the way K is summed is a
function of the shape alone."""
import pytest

from aginfer_b200.recipes.builder import TC_SCRATCH_BYTES, TK_CLUSTERS, k_runs, tk_tiling

SHAPES = [(16, 128), (130, 256), (2048, 2048), (11008, 2048), (2048, 11008), (3584, 18944), (151, 640)]


@pytest.mark.parametrize("M", [33, 64, 65, 127, 128, 129, 288, 513, 1024])
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
