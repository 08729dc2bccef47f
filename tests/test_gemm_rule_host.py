"""The tensor-core GEMM's pipeline depth (openhurricane_b200/csrc/gemm_rule.h) compiled for
the host: the short ring only for a short K and where two blocks can share an SM, that is, where
the grid has more blocks than the GPU has SMs."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_short_ring_only_for_grids_beyond_the_sms(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "rule")
    subprocess.check_call([gxx, "-O1", "-std=c++17", "-o", exe, os.path.join(HERE, "cpp", "gemm_rule.cpp")])
    # a training batch's layers and weight gradients (K = batch); an inference chunk; the
    # edges of 148 SMs and of a short K; a grid beyond 32 bits
    cases = [((1, 1, 256, 148), 4), ((4, 1, 256, 148), 4), ((2, 1, 512, 148), 4), ((64, 1, 256, 148), 4),
             ((64, 2, 256, 148), 4), ((74, 2, 256, 148), 4), ((149, 1, 64, 148), 2), ((512, 1, 256, 148), 2),
             ((512, 1, 512, 148), 2), ((512, 1, 576, 148), 4), ((100000, 100000, 256, 148), 2)]
    txt = "\n".join(" ".join(map(str, c)) for c, _ in cases)
    out = subprocess.run([exe], input=txt, capture_output=True, text=True, check=True).stdout.split()
    assert [int(v) for v in out] == [w for _, w in cases]
