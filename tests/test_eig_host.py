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


@pytest.mark.parametrize("op,lo,bound", [("tan", 1.0, 2.0 ** -50), ("tandf", 0.5, 2.0 ** -44)])
def test_rotation_angle(harness, op, lo, bound):
    """The rotation's tangent against r t^2 + d t - r = 0 solved in 60 digits: an eigenvector is as good as its last
    rotations, so the angle is rounding in its own arithmetic (FP64: two Newton steps end at a residual of some 3 roundings
    of r over a slope >= 2 r; double-float: one step from 2^-23 leaves 2^-46 and its operations 2^-45)."""
    from decimal import Decimal as Dc, getcontext
    getcontext().prec = 60
    rng = np.random.default_rng(11)
    cases = []
    for i in range(600):
        r = rng.uniform(lo, 1.4 * 2 * lo)
        d = float(np.exp(rng.uniform(-40, 30)) * rng.choice([-1, 1])) if i % 3 else float(rng.normal() * r)
        if op == "tandf":
            r, d = [(float(np.float32(x)), float(np.float32(x - float(np.float32(x))))) for x in (r, d)]
            cases.append((r[0], r[1], d[0], d[1]))
        else:
            cases.append((r, d))
    cases.append((1.25, 0.0) if op == "tan" else (1.25, 0.0, 0.0, 0.0))
    out = harness(["%s %s\n" % (op, " ".join(x.hex() for x in c)) for c in cases])
    for c, o in zip(cases, out):
        r, d = (Dc(c[0]), Dc(c[1])) if op == "tan" else (Dc(c[0]) + Dc(c[1]), Dc(c[2]) + Dc(c[3]))
        t = sum((Dc(float.fromhex(x)) for x in o), Dc(0))
        exact = 2 * r / (abs(d) + (d * d + 4 * r * r).sqrt()) * (1 if d >= 0 else -1)
        assert abs(t - exact) <= Dc(bound) * abs(exact)
