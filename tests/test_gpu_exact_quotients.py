"""Quotients by a corrected reciprocal beside the divisions they stand for: SwiGLU over every bf16 gate, E4M3 quantisation of
every bf16 value for every bf16 amax."""
import subprocess
from pathlib import Path

import pytest
import torch

from aginfer_b200.build import KERNEL_SRC, nvcc
from aginfer_b200.recipes import Tensor, U32, package
from oracle import ops
from tests.gpu_util import run_recipe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
EVERY = torch.arange(65536, dtype=torch.int32).to(torch.uint16).view(BF)


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    cubin = tmp_path_factory.mktemp("probe") / "kernels.cubin"
    subprocess.run([nvcc(), "-cubin", "-arch=sm_100a", "-O3", "-std=c++17", f"-I{KERNEL_SRC}", "-o", str(cubin),
                    str(Path(__file__).with_name("quotient_probe.cu"))], check=True)
    return cubin


def test_silu_of_every_gate_is_the_divisions_in_fp32(tmp_path, probe, monkeypatch):
    monkeypatch.setattr(package, "CUBIN", probe)

    def body(r):
        r.launch("probe_silu_f32", (64, 1, 1), (256, 1, 1), [Tensor("x"), Tensor("got"), Tensor("want"), U32(65536)])

    out, _ = run_recipe(tmp_path, {}, {"x": EVERY}, {n: (torch.float32, (65536,)) for n in ("got", "want")}, body)
    got, want = out["got"], out["want"]
    differ = (got.view(torch.int32) != want.view(torch.int32)) & ~(got.isnan() & want.isnan())
    assert not differ.any(), [(x, g, w) for x, g, w in zip(EVERY[differ].tolist()[:8], got[differ].tolist(), want[differ].tolist())]


def test_e4m3_codes_of_every_value_for_every_amax_are_the_divisions(tmp_path, probe, monkeypatch):
    monkeypatch.setattr(package, "CUBIN", probe)
    count = 0x7f80 + 1                          # 0, every finite amax and infinity

    def body(r):
        r.launch("probe_e4m3_codes", (count, 1, 1), (256, 1, 1), [Tensor("differ"), U32(0)])

    out, _ = run_recipe(tmp_path, {}, {"x": EVERY[:8]}, {"differ": (torch.int32, (count,))}, body)
    assert not out["differ"].any(), out["differ"].nonzero().flatten().tolist()[:8]


def test_swiglu_of_every_gate_equals_the_silu_that_divides(tmp_path):
    def body(r):
        r.swiglu(Tensor("gate"), Tensor("one"), Tensor("y"), 64, 1024, 1024)
        r.launch("agi_silu_bf16", (256, 1, 1), (256, 1, 1), [Tensor("gate"), Tensor("want"), U32(65536)])

    got, _ = run_recipe(tmp_path, {}, {"gate": EVERY, "one": torch.ones(65536, dtype=BF)},
                        {"y": (BF, (65536,)), "want": (BF, (65536,))}, body)
    same = got["y"].view(torch.int16) == got["want"].view(torch.int16)
    assert (same | (got["y"].isnan() & got["want"].isnan())).all()


@pytest.mark.parametrize("exponent", [-126, -100, -79, -78, -72, -71, -20, 0, 7, 60, 87, 88, 89, 90, 127])
@pytest.mark.parametrize("mantissa", [1.0, 1.3359375, 1.9921875])
def test_quantisation_of_every_value_up_to_amax(tmp_path, exponent, mantissa):
    amax = torch.tensor(mantissa * 2.0 ** exponent, dtype=BF)
    x = torch.where(EVERY.abs() <= amax, EVERY, amax)       # NaN: amax

    def body(r):
        r.quantize_e4m3(Tensor("x"), Tensor("q"), r.alloc(4), 65536)

    got, _ = run_recipe(tmp_path, {}, {"x": x}, {"q": (torch.float8_e4m3fn, (65536,))}, body)
    want, _ = ops.quantize_e4m3(x)
    assert torch.equal(got["q"].view(torch.uint8), want.view(torch.uint8))
