"""Host checks of the lattice kernels' own source (dmftpack_gb300/csrc/schur.cuh, df.cuh, compiled for the host by nvcc)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("lattice") / "lattice_check")
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a", "-Xcompiler",
                        "-ffp-contract=off", "-I", os.path.join(ROOT, "include"), "-I",
                        os.path.join(ROOT, "dmftpack_gb300", "csrc"), os.path.join(ROOT, "tests", "cxx", "lattice_check.cu"),
                        "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(lines):
        out = subprocess.run([exe], input="".join(lines), capture_output=True, text=True, timeout=120)
        assert out.returncode == 0, out.stderr
        return [ln.split() for ln in out.stdout.splitlines()]
    return run


@pytest.mark.parametrize("untuned", [4, 8, 16, 24])
def test_autotuner_times_the_untuned_launch(harness, untuned):
    c = [int(x) for x in harness(["cps %d\n" % untuned])[0]]
    assert c[0] == untuned and len(set(c)) == len(c) and {4, 8, 16} <= set(c)
