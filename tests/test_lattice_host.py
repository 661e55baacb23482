"""Host checks of the lattice kernels' own source (dmftpack_gb300/csrc/schur.cuh, df.cuh, compiled for the host by nvcc)."""
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


def _line(op, M):
    return "%s %s\n" % (op, " ".join("%s %s" % (float(z.real).hex(), float(z.imag).hex()) for z in np.ravel(M)))


def test_two_by_two_inverse(harness):
    """The closed form of the 2 x 2 inverse: singular matrices whose products are equal (rows alike, zero rows, powers of two)
    are flagged, also where the products round; z - H - Sigma is inverted to a few roundings times its condition."""
    rng = np.random.default_rng(4)
    sing = [np.zeros((2, 2)), np.array([[1.0, 0], [0, 0]]), np.array([[0, 0], [0.3, 2j]])]
    for c in rng.normal(size=40):
        sing += [np.full((2, 2), c), np.array([[c, 2 * c], [c, 2 * c]]), np.array([[c, -c], [4 * c, -4 * c]]) * 1j]
    assert all(r[0] == "1" for r in harness([_line("inv2d", M) for M in sing]))
    good = []
    for _ in range(300):
        H = rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2))
        good.append((rng.normal() + 1j * np.exp(rng.uniform(-4, 4))) * np.eye(2) - (H + H.conj().T) / 2)
    for M, r in zip(good, harness([_line("inv2d", M) for M in good])):
        v = np.array([float.fromhex(x) for x in r[1:]])
        X, exact = (v[0::2] + 1j * v[1::2]).reshape(2, 2), np.linalg.inv(M)
        assert r[0] == "0" and np.abs(X - exact).max() <= 16 * 2.0 ** -53 * np.linalg.cond(M) * np.abs(exact).max()


def _split(x):
    h = float(np.float32(x))
    return h, float(np.float32(x - h))


def test_packed_arithmetic_has_the_scalar_bits(harness):
    """OpsP, which the lattice and eigensolver kernels compute in, against OpsF, whose operations are held to exact rational
    arithmetic: the same bits."""
    rng = np.random.default_rng(9)
    lines = []
    for _ in range(500):
        d = [_split(float(x)) for x in np.exp(rng.uniform(-8, 8, 6)) * rng.choice([-1, 1], 6)]
        lines.append("pack %s\n" % " ".join(x.hex() for hl in d for x in hl))
    assert all(r == ["0"] * 6 for r in harness(lines))


@pytest.mark.parametrize("n", [2, 3])
def test_packed_inverse(harness, n):
    """The 2 x 2 closed form and the 3 x 3 elimination of the thread-per-frequency kernels in packed double-float: z - H - Sigma
    over the energies a determinant in FP32's range allows, and rows in other orders; within 2^-44 of the entries' scale
    times the condition, as the scalar form is held to."""
    rng = np.random.default_rng(n)
    mats = []
    for t in range(300):
        H = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
        M = (0.3 + 1j * np.exp(rng.uniform(-3, 2))) * np.eye(n) - (H + H.conj().T) / 2
        M = M[rng.permutation(n)] * 10.0 ** rng.integers(-8, 9)
        mats.append(np.array([complex(sum(_split(z.real)), sum(_split(z.imag))) for z in M.ravel()]).reshape(n, n))
    for M, r in zip(mats, harness([_line("inv%dp" % n, M) for M in mats])):
        v = np.array([float.fromhex(x) for x in r[1:]])
        X, exact = (v[0::2] + 1j * v[1::2]).reshape(n, n), np.linalg.inv(M)
        assert r[0] == "0" and np.abs(X - exact).max() <= 2.0 ** -44 * np.linalg.cond(M) * np.abs(exact).max()


def test_reciprocal_root(harness):
    from decimal import Decimal as Dc, getcontext
    getcontext().prec = 50
    rng = np.random.default_rng(6)
    xs = [_split(float(x)) for x in np.exp(rng.uniform(-20, 20, 300))]
    for x, r in zip(xs, harness(["rsqrt %s %s\n" % (a.hex(), b.hex()) for a, b in xs])):
        exact = 1 / (Dc(x[0]) + Dc(x[1])).sqrt()
        assert abs(Dc(float.fromhex(r[0])) + Dc(float.fromhex(r[1])) - exact) <= Dc(2.0 ** -44) * exact
