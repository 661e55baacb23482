"""Host checks of the per-k eigensolver's own source (dmftpack_gb300/csrc/eig.cuh, compiled for the host by nvcc)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("eig") / "eig_check")
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a", "-Xcompiler",
                        "-ffp-contract=off", "-I", os.path.join(ROOT, "include"), "-I",
                        os.path.join(ROOT, "dmftpack_gb300", "csrc"), os.path.join(ROOT, "tests", "cxx", "eig_check.cu"),
                        "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(lines):
        out = subprocess.run([exe], input="".join(lines), capture_output=True, text=True, timeout=120)
        assert out.returncode == 0, out.stderr
        return [ln.split() for ln in out.stdout.splitlines()]
    return run


def test_order_of_eigenvalues_is_a_permutation(harness):
    """The order addresses the eigenvectors: it has to be a permutation for any values, NaN, infinities and ties among
    them, ascending with NaN last."""
    rng = np.random.default_rng(2)
    cases = [[float("nan")], [float("nan")] * 28, [1.0, float("nan"), 1.0, float("-inf"), float("inf"), float("nan"), -0.0, 0.0]]
    for n in (2, 5, 12, 64):
        for bad in (0, 1, n // 2, n):
            w = rng.integers(-3, 4, size=n).astype(float)
            w[rng.permutation(n)[:bad]] = rng.choice([np.nan, np.inf, -np.inf], size=bad)
            cases.append(list(w))
    out = harness(["rank %d %s\n" % (len(w), " ".join("nan" if np.isnan(x) else float(x).hex() for x in w)) for w in cases])
    for w, r in zip(cases, out):
        rank = np.array([int(x) for x in r])
        assert sorted(rank) == list(range(len(w)))
        assert np.array_equal(np.array(w)[np.argsort(rank)], np.sort(w), equal_nan=True)
