"""The host side of the C ABI against a CUDA runtime made up in host_logic.cpp: orders of
calls by two callers, calls that fail, plans, which no GPU is needed for and which a GPU would
meet by chance."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mlx-data_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
SOURCES = ["context.cu", "api.cu", "launch_plan.cu", "noalloc.cu"]


def build(tmp_path_factory, *flags):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and CUDA's headers")
    out = str(tmp_path_factory.mktemp("host_logic") / "host_logic")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", *flags, "-I" + os.path.join(CUDA, "include"), "-I" + CSRC,
                    "-x", "c++", os.path.join(HERE, "host_logic.cpp")] +
                   [os.path.join(CSRC, s) for s in SOURCES] + ["-o", out], check=True)
    return out


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    return build(tmp_path_factory)


@pytest.fixture(scope="module")
def plain_program(tmp_path_factory):
    # as on a host without SSE2: no intrinsics, their headers empty
    return build(tmp_path_factory, "-U__SSE2__", "-D_EMMINTRIN_H_INCLUDED", "-D_XMMINTRIN_H_INCLUDED")


@pytest.mark.parametrize("scenario", ["wait_beside_another_caller", "copies_of_huge_sources_beside_a_resize",
                                      "failed_copy_of_a_part", "timed_calls_take_the_same_way",
                                      "casts_with_nan_keep_the_table", "casts_without_a_cache", "packed_sources"])
def test_scenario(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout + r.stderr)


@pytest.mark.parametrize("scenario", ["packed_sources", "wait_beside_another_caller"])
def test_without_sse2(plain_program, scenario):
    r = subprocess.run([plain_program, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout + r.stderr)
