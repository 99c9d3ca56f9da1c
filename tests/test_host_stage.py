"""The operator face's host side built by itself against fakes of the CUDA calls it makes: conversions (both the vector forms and
the plain loops other hosts run), the piece pipeline, and its behaviour when a call fails."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tpu-mlir_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

pytestmark = pytest.mark.skipif(shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")),
                                reason="needs g++ and the CUDA headers")


@pytest.fixture(scope="module", params=["vector", "plain"])
def program(request, tmp_path_factory):
    out = str(tmp_path_factory.mktemp("host_stage") / "check")
    cmd = ["g++", "-O2", "-std=c++17", "-Wall", "-Wno-unused-function", "-ffp-contract=off", "-pthread", "-I" + CSRC, "-I" + os.path.join(CUDA, "include"),
           os.path.join(ROOT, "tests", "host_stage_check.cpp"), os.path.join(CSRC, "host_convert.cpp"),
           os.path.join(CSRC, "host_stage.cpp"), "-o", out, "-ldl"]
    if request.param == "plain":
        cmd.append("-DB200Q_PORTABLE_HOST")
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("what", ["conversions", "pieces", "no threads", "two threads", "out of memory", "streams", "copies", "overlap", "held arrays", "workers"])
def test_host_stage(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr


def test_vector_code_is_for_x86_hosts_only():
    for name in os.listdir(CSRC):
        if name.endswith((".cpp", ".h", ".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            if "immintrin.h" in text or "_mm_pause" in text:
                assert name == "host_convert.cpp" and text.index("defined(__x86_64__)") < text.index("immintrin.h")
