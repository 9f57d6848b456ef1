"""Which CTA walks which span (lasp_b200/csrc/span_cut.h), simulated on the CPU with the header the kernels use."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def sim(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("cutsim") / "span_cut_sim")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "lasp_b200", "csrc"),
                           os.path.join(ROOT, "tests", "csrc", "span_cut_sim.cpp"), "-o", exe])
    return exe


@pytest.mark.parametrize("sms", [132, 148, 160])
def test_every_tile_once_and_waits_for_earlier_ctas_only(sim, sms):
    out = subprocess.run([sim, str(sms)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
