"""Kernels called through the library's launchers by tests/host_cpp/kernels.cu (built here with nvcc), against sums in 64 bits."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def kernels(pkg, tmp_path_factory):
    out = str(tmp_path_factory.mktemp("kernels") / "kernels")
    lib = pkg.library_path()
    r = subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-I", os.path.join(os.path.dirname(lib), "csrc"),
                        os.path.join(ROOT, "tests", "host_cpp", "kernels.cu"), "-o", out, lib, "-Xlinker", "-rpath", "-Xlinker", os.path.dirname(lib)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("check", ["attention-sums", "attention-specials", "attention-prompt", "attention-band", "experts", "matvec-bf16", "matvec-q8", "matvec-peer", "few-rows", "gave-up", "level-specials", "claims"])
def test_kernels(kernels, check):
    r = subprocess.run([kernels, check], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
