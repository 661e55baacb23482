"""GPU parity of the lattice stage (H(k), G_loc, N(mu), mu search, Delta, moments) against the FP64 oracle.
Every call goes through the C ABI (libdmftgpu.so via ctypes)."""
import numpy as np
import pytest

from conftest import rel_err
from dmftpack_gb300 import lib, models

pytestmark = pytest.mark.gpu

TOL = 1e-10   # relative, plain FP64 path vs FP64 oracle
TOL_MIXED = 1e-9   # double-float (split-precision) path vs FP64 oracle


def _setup(orc, wl):
    km = orc.kmesh(*wl.kgrid)
    H = orc.hk(wl.n, wl.rindex, wl.hr, km)
    lat = lib.Lattice(wl.n, wl.nk, wl.nfreq, wl.beta, wl.ncl, wl.nh)
    return H, lat


def test_hk_matches_oracle(ctx, orc):
    wl = models.t2g_p(k=5, nfreq=16)
    H = orc.hk(wl.n, wl.rindex, wl.hr, orc.kmesh(*wl.kgrid))
    Hg = ctx.Construct_Hk(wl.n, wl.rindex, wl.hr, wl.kgrid)
    assert rel_err(Hg, H) < 1e-13
    import torch
    Hd = ctx.Construct_Hk(wl.n, wl.rindex, wl.hr, wl.kgrid, device_out=torch.device("cuda:0"))
    assert rel_err(Hd.cpu().numpy(), H) < 1e-13


@pytest.mark.parametrize("mixed", [False, True])
def test_hk_rows_in_any_order(ctx, orc, mixed):
    """Rows of one lattice vector that do not follow each other, repeated rows, a table larger than the previous one."""
    rng = np.random.default_rng(5)
    for n, nvec in ((2, 3), (5, 27)):
        R = rng.integers(-3, 4, size=(nvec, 3))
        rows = np.concatenate([R[rng.integers(0, nvec, 40 * nvec)], rng.integers(0, n, size=(40 * nvec, 2))], 1).astype(np.int32)
        hr = rng.normal(size=len(rows)) + 1j * rng.normal(size=len(rows))
        H = orc.hk(n, rows, hr, orc.kmesh(3, 4, 5))
        assert rel_err(ctx.Construct_Hk(n, rows, hr, (3, 4, 5), mixed=mixed), H) < (1e-10 if mixed else 1e-13)


@pytest.mark.parametrize("case", ["t2g_p", "dp28", "soc56", "hubbard"])
def test_hk_tensor_cores_match_oracle(ctx, orc, case):
    """H(k) as a tcgen05 GEMM (bf16 slices, exact level sums): k counts and 2 n^2 that are not multiples of the
    128 x 48 tile, N_R = 9 .. 729, against the FP64 oracle at the plain form's tolerance; a second call reuses
    the cached phase image."""
    wl = {"t2g_p": lambda: models.t2g_p(k=5, nfreq=8), "dp28": lambda: models.dp28(k=3, nfreq=8, ntau=16),
          "soc56": lambda: models.soc56(k=3, nfreq=8), "hubbard": lambda: models.hubbard_2d(kx=11, ky=13, nfreq=8)}[case]()
    H = orc.hk(wl.n, wl.rindex, wl.hr, orc.kmesh(*wl.kgrid))
    for _ in range(2):
        Ht = ctx.Construct_Hk(wl.n, wl.rindex, wl.hr, wl.kgrid, mixed=True)
        assert rel_err(Ht, H) < TOL


@pytest.mark.parametrize("green", [False, True])
def test_moments_match_oracle(ctx, orc, green):
    wl = models.t2g_p(k=2, nfreq=200, beta=20.0)
    F = wl.sigma if not green else np.linalg.inv(1j * wl.wn()[:, None, None] * np.eye(3)[None]
                                                   - 0.3 * np.eye(3)[None] - wl.sigma)
    m_o = orc.moments(F, wl.beta, green_asym=green)
    m_g = ctx.getAsymto_moments(F, wl.beta, greenFtnAsym=green)
    for i in range(4):
        assert np.abs(m_g[i] - m_o[i]).max() <= 1e-9 * max(1.0, np.abs(m_o[i]).max()), i


CASES = {
    "t2g_p": lambda: models.t2g_p(k=4, nfreq=40, beta=12.0),
    "hubbard": lambda: models.hubbard_2d(kx=8, ky=8, nfreq=48, beta=10.0),
}


@pytest.mark.gpu
@pytest.mark.parametrize("D,nf,green", [(1, 20, False), (2, 33, False), (7, 64, False), (20, 65, False), (33, 40, False),
                                        (46, 24, False), (2, 12900, False), (1, 20, True), (11, 97, True),
                                        (46, 24, True), (1, 12900, True)])
def test_moments_edges(ctx, orc, D, nf, green):
    """Smallest and ragged N_freq, N_freq beyond the staged sums, matrices beyond the gates' shared memory.  The moments
    describe the tail beyond the data: it is compared there, relative to its size.  Bound: the fits' 2 x 2 normal
    matrices over a window of a tenth of the axis amplify the rounding of sums of nf terms by ~1e3: 2e-16 1e3 sqrt(nf)
    < 2e-11, with a factor 5 for the extrapolation."""
    rng = np.random.default_rng([D, nf])
    w = np.pi * (2 * np.arange(nf) + 1) / 30.0
    if green:
        A = rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D))
        F = np.linalg.inv(1j * w[:, None, None] * np.eye(D) - (A + A.conj().T) / (2 * np.sqrt(D)))
    else:
        F = np.zeros((nf, D, D), complex)
        F[:, np.arange(D), np.arange(D)] = -1j * rng.uniform(0.4, 0.6, D) / (w[:, None] + rng.uniform(0.8, 1.2, D))
    x = 1j * np.pi * (2 * np.array([nf, 2 * nf, 4 * nf]) + 1) / 30.0
    tail = lambda m: sum(m[i][None] / x[:, None, None] ** i for i in range(4))
    a, b = tail(ctx.getAsymto_moments(F, 30.0, greenFtnAsym=green)), tail(orc.moments(F, 30.0, green_asym=green))
    for p, q in zip(a, b):
        assert np.abs(p - q).max() <= 1e-10 * np.abs(q).max()


@pytest.mark.parametrize("explicit", [False, True])
@pytest.mark.parametrize("case", list(CASES))
def test_greenftn_w_matches_oracle(ctx, orc, case, explicit):
    wl = CASES[case]()
    H, lat = _setup(orc, wl)
    mu = 0.25
    gw, gwhf, num = orc.greenftn_w(H, wl.sigma, mu, wl.beta, wl.ncl, wl.nh)
    g_gw, g_gwhf, g_num = ctx.GreenFtn_w(lat, H, wl.sigma, mu, explicit=explicit)
    assert rel_err(g_gw, gw) < TOL
    assert rel_err(g_gwhf, gwhf) < TOL
    assert rel_err(g_num, num) < TOL


def test_greenftn_w_device_pointers(ctx, orc):
    import torch
    wl = CASES["t2g_p"]()
    H, lat = _setup(orc, wl)
    gw, gwhf, num = orc.greenftn_w(H, wl.sigma, 0.1, wl.beta, wl.ncl, wl.nh)
    dev = torch.device("cuda:0")
    g_gw, g_gwhf, g_num = ctx.GreenFtn_w(lat, torch.from_numpy(H).to(dev), torch.from_numpy(wl.sigma).to(dev), 0.1)
    torch.cuda.synchronize()
    assert rel_err(g_gw.cpu().numpy(), gw) < TOL
    assert rel_err(g_num.cpu().numpy(), num) < TOL


@pytest.mark.parametrize("explicit", [False, True])
@pytest.mark.parametrize("n,D,hartr", [(5, 2, [3, 1]), (7, 3, None), (3, 1, [2]), (16, 5, None), (9, 9, None)])
def test_greenftn_w_padding_and_hartree_index(ctx, orc, n, D, hartr, explicit):
    """Odd sizes (identity padding to the next instantiated N) and a HartrIndex that is not the identity."""
    rng = np.random.default_rng(n * 10 + D)
    nk, nf, beta = 27, 32, 8.0
    A = rng.normal(size=(nk, n, n)) + 1j * rng.normal(size=(nk, n, n))
    H = (A + np.conj(np.swapaxes(A, 1, 2))) / 2
    wn = np.pi * (2 * np.arange(nf) + 1) / beta
    S = np.zeros((nf, D, D), complex)
    for d in range(D):
        S[:, d, d] = 0.2 - 0.7j / (wn + 0.5)
    h = np.arange(D) if hartr is None else np.array(hartr)
    lat = lib.Lattice(n, nk, nf, beta, 1, D, hartr=h)
    gw, gwhf, num = orc.greenftn_w(H, S, -0.3, beta, 1, D, hartr=h)
    g_gw, g_gwhf, g_num = ctx.GreenFtn_w(lat, H, S, -0.3, explicit=explicit)
    assert rel_err(g_gw, gw) < TOL and rel_err(g_gwhf, gwhf) < TOL and rel_err(g_num, num) < TOL
    N, dN = orc.nele(H, S, -0.3, beta, 1, D, hartr=h, deriv=True)
    gN, gdN = ctx.GiwToNele(lat, H, S, -0.3, deriv=True, explicit=explicit)
    assert abs(gN - N) < 1e-11 * max(1, abs(N)) and abs(gdN - dN) < 1e-9 * abs(dN)


@pytest.mark.parametrize("n,D,hartr", [(5, 2, [3, 1]), (7, 3, None), (12, 3, None), (16, 5, None), (9, 9, None),
                                        (28, 10, None)])
def test_explicit_mixed_matches_oracle(ctx, orc, n, D, hartr):
    """The reference's own algorithm (an explicit n x n inversion of every (k, iw) matrix, src/GreenFtn.cpp:245-261)
    in double-float on the FP32 pipe (DMFTGPU_EXPLICIT | DMFTGPU_MIXED): G_loc, GwHF, NumMatrix, N and dN/dmu."""
    rng = np.random.default_rng(n * 7 + D)
    nk, nf, beta = 27, 32, 8.0
    A = rng.normal(size=(nk, n, n)) + 1j * rng.normal(size=(nk, n, n))
    H = (A + np.conj(np.swapaxes(A, 1, 2))) / 2
    wn = np.pi * (2 * np.arange(nf) + 1) / beta
    S = np.zeros((nf, D, D), complex)
    for d in range(D):
        S[:, d, d] = 0.2 - 0.7j / (wn + 0.5)
    S[:, 0, D - 1] = S[:, D - 1, 0] = 0.05 if D > 1 else 0
    h = np.arange(D) if hartr is None else np.array(hartr)
    lat = lib.Lattice(n, nk, nf, beta, 1, D, hartr=h)
    gw, gwhf, num = orc.greenftn_w(H, S, -0.3, beta, 1, D, hartr=h)
    g_gw, g_gwhf, g_num = ctx.GreenFtn_w(lat, H, S, -0.3, explicit=True, mixed=True)
    assert rel_err(g_gw, gw) < TOL_MIXED and rel_err(g_gwhf, gwhf) < TOL_MIXED and rel_err(g_num, num) < TOL_MIXED
    N, dN = orc.nele(H, S, -0.3, beta, 1, D, hartr=h, deriv=True)
    gN, gdN = ctx.GiwToNele(lat, H, S, -0.3, deriv=True, explicit=True, mixed=True)
    assert abs(gN - N) < 1e-10 * max(1, abs(N)) and abs(gdN - dN) < 1e-9 * abs(dN)


def test_large_orbital_count_schur_only(ctx, orc):
    """n = 56 with a 20-orbital correlated block (beyond the explicit kernels' register budget)."""
    rng = np.random.default_rng(5)
    n, D, nk, nf, beta = 56, 20, 8, 24, 5.0
    A = rng.normal(size=(nk, n, n)) + 1j * rng.normal(size=(nk, n, n))
    H = (A + np.conj(np.swapaxes(A, 1, 2))) / 4
    wn = np.pi * (2 * np.arange(nf) + 1) / beta
    S = np.zeros((nf, D, D), complex)
    for d in range(D):
        S[:, d, d] = -0.4j / (wn + 0.7)
    lat = lib.Lattice(n, nk, nf, beta, 1, D)
    gw, gwhf, num = orc.greenftn_w(H, S, 0.1, beta, 1, D)
    g_gw, g_gwhf, g_num = ctx.GreenFtn_w(lat, H, S, 0.1)
    assert rel_err(g_gw, gw) < TOL and rel_err(g_gwhf, gwhf) < TOL and rel_err(g_num, num) < TOL


def test_two_clusters(ctx, orc):
    rng = np.random.default_rng(11)
    n, nk, nf, beta, ncl, nh = 8, 16, 32, 6.0, 2, 2
    A = rng.normal(size=(nk, n, n)) + 1j * rng.normal(size=(nk, n, n))
    H = (A + np.conj(np.swapaxes(A, 1, 2))) / 2
    wn = np.pi * (2 * np.arange(nf) + 1) / beta
    S = np.zeros((nf, 4, 4), complex)
    for d in range(4):
        S[:, d, d] = -0.3j / (wn + 1)
    lat = lib.Lattice(n, nk, nf, beta, ncl, nh)
    gw, gwhf, num = orc.greenftn_w(H, S, 0.0, beta, ncl, nh)
    for explicit in (False, True):
        g_gw, g_gwhf, g_num = ctx.GreenFtn_w(lat, H, S, 0.0, explicit=explicit)
        assert rel_err(g_gw, gw) < TOL and rel_err(g_num, num) < TOL
        N = orc.nele(H, S, 0.0, beta, ncl, nh)
        assert abs(ctx.GiwToNele(lat, H, S, 0.0, explicit=explicit) - N) < 1e-11 * abs(N)


@pytest.mark.parametrize("explicit", [False, True])
@pytest.mark.parametrize("case", list(CASES))
def test_nele_matches_oracle(ctx, orc, case, explicit):
    wl = CASES[case]()
    H, lat = _setup(orc, wl)
    for mu in (-0.5, 0.25):
        N, dN = orc.nele(H, wl.sigma, mu, wl.beta, wl.ncl, wl.nh, deriv=True)
        gN, gdN = ctx.GiwToNele(lat, H, wl.sigma, mu, deriv=True, explicit=explicit)
        assert abs(gN - N) < 1e-11 * max(1, abs(N))
        assert abs(gdN - dN) < 1e-9 * abs(dN)


def test_adjust_mu_bisection_matches_oracle_and_newton_converges(ctx, orc):
    wl = CASES["t2g_p"]()
    H, lat = _setup(orc, wl)
    target = 7.3
    mu_o, ne_o = orc.adjust_mu(H, wl.sigma, 0.0, wl.beta, wl.ncl, wl.nh, target)
    mu_g, ne_g = ctx.GreenFtn_w_adjust_mu(lat, H, wl.sigma, 0.0, 1.0, target)
    assert ne_g == ne_o and abs(mu_g - mu_o) <= 1e-12
    mu_x, ne_x = ctx.GreenFtn_w_adjust_mu(lat, H, wl.sigma, 0.0, 1.0, target, explicit=True)
    assert ne_x == ne_o and abs(mu_x - mu_o) <= 1e-12
    mu_n, ne_n = ctx.GreenFtn_w_adjust_mu(lat, H, wl.sigma, 0.0, 1.0, target, newton=True)
    assert abs(mu_n - mu_o) < 2e-5
    assert abs(orc.nele(H, wl.sigma, mu_n, wl.beta, wl.ncl, wl.nh) - target) < 1e-9
    assert ne_n < ne_o


def _random_lattice(n, D, kgrid, nf, seed):
    rng = np.random.default_rng(seed)
    nk = kgrid[0] * kgrid[1] * kgrid[2]
    A = rng.normal(size=(nk, n, n)) + 1j * rng.normal(size=(nk, n, n))
    H = (A + A.conj().transpose(0, 2, 1)) / 2
    w = np.pi * (2 * np.arange(nf) + 1) / 15.0
    S = np.zeros((nf, D, D), complex)
    S[:, np.arange(D), np.arange(D)] = -1j * rng.uniform(0.4, 0.6, D) / (w[:, None] + rng.uniform(0.8, 1.2, D))
    return H, S, lib.Lattice(n, nk, nf, 15.0, 1, D)


@pytest.mark.parametrize("n,D,kgrid,nf", [(1, 1, (3, 1, 1), 24), (2, 1, (5, 3, 1), 64), (2, 2, (7, 1, 1), 65),
                                          (3, 2, (3, 3, 1), 24), (3, 3, (9, 1, 1), 24), (9, 3, (17, 1, 1), 70),
                                          (40, 3, (2, 2, 2), 24), (33, 2, (3, 1, 1), 129)])
def test_nele_small_blocks(ctx, orc, n, D, kgrid, nf):
    """N(mu) and dN/dmu of correlated blocks up to 3 x 3 (one thread per frequency): without ligands, with one and with
    more poles than a renormalisation run, k counts around the staging and chunk sizes, ragged frequency tiles; bounds
    of the other N(mu) tests (FP64 1e-11, double-float 1e-9)."""
    H, S, lat = _random_lattice(n, D, kgrid, nf, [n, D, nf])
    for mu in (-0.4, 0.3):
        N, dN = orc.nele(H, S, mu, 15.0, 1, D, deriv=True)
        for mixed, tol in ((False, 1e-11), (True, 1e-9)):
            g, dg = ctx.GiwToNele(lat, H, S, mu, deriv=True, mixed=mixed)
            assert abs(g - N) <= tol * max(1, abs(N)) and abs(dg - dN) <= 10 * tol * max(1, abs(dN))
            assert abs(ctx.GiwToNele(lat, H, S, mu, mixed=mixed) - N) <= tol * max(1, abs(N))


@pytest.mark.parametrize("newton", [False, True])
def test_adjust_mu_reports_singular_inversion(ctx, newton):
    """A zero pivot inside the mu search is reported as SINGULAR by both search modes (the reference would
    carry inf/nan on silently).  Flat band H(k) = 0 and Sigma(i w_0) = mu0 + i w_0 make z - H - Sigma exactly
    zero at the first frequency for the first mu evaluated."""
    nk, nf, beta, mu0 = 8, 16, 10.0, 0.3
    H = np.zeros((nk, 1, 1), complex)
    wn = np.pi * (2 * np.arange(nf) + 1) / beta
    S = (-0.5j / (wn + 1.0)).reshape(nf, 1, 1).astype(complex)
    S[0, 0, 0] = complex(mu0, np.pi / beta)
    lat = lib.Lattice(1, nk, nf, beta, 1, 1)
    with pytest.raises(lib.DmftGpuError) as e:
        ctx.GreenFtn_w_adjust_mu(lat, H, S, mu0, 1.0, 0.5, newton=newton)
    assert e.value.code == lib.SINGULAR




@pytest.mark.parametrize("n,D,nf", [(12, 4, 40), (16, 6, 33), (20, 8, 48), (28, 10, 64), (19, 9, 40), (40, 10, 24),
                                    (11, 5, 16)])
def test_nele_tensor_cores_match_oracle(ctx, orc, n, D, nf):
    """N(mu) with the pole sums on the tensor cores (bf16 slices, exact top levels) and the inversions in
    double-float: block widths 4 .. 10 (padded ones included), m = n - D up to 30, frequency counts that leave a
    partial 32-frequency tile.  Against the FP64 oracle with a diagonal Sigma, and, with an off-diagonal Sigma
    element added, against the GPU's FP64 and CUDA-core double-float passes (the same tail moments on every path:
    for that Sigma the moment fit's window choice compares variances that are equal up to rounding, so the
    oracle may pick another window)."""
    rng = np.random.default_rng(100 * n + D)
    nk, beta = 27, 8.0
    A = rng.normal(size=(nk, n, n)) + 1j * rng.normal(size=(nk, n, n))
    H = (A + np.conj(np.swapaxes(A, 1, 2))) / 3
    wn = np.pi * (2 * np.arange(nf) + 1) / beta
    S = np.zeros((nf, D, D), complex)
    for d in range(D):
        S[:, d, d] = 0.1 * d - 0.6j / (wn + 0.4)
    lat = lib.Lattice(n, nk, nf, beta, 1, D)
    for mu in (-0.4, 0.3):
        N = orc.nele(H, S, mu, beta, 1, D)
        gN = ctx.GiwToNele(lat, H, S, mu, mixed=True)
        assert abs(gN - N) < TOL_MIXED * max(1.0, abs(N)), (gN, N)
    S[:, 0, 1] = S[:, 1, 0] = 0.05 / (1j * wn + 1.0)
    for mu in (-0.4, 0.3):
        gF = ctx.GiwToNele(lat, H, S, mu)
        gN = ctx.GiwToNele(lat, H, S, mu, mixed=True)
        gC = ctx.GiwToNele(lat, H, S, mu, mixed=True, tensor=False)
        assert abs(gN - gF) < 1e-11 * max(1.0, abs(gF)), (gN, gF)
        assert abs(gC - gF) < 1e-11 * max(1.0, abs(gF)), (gC, gF)


@pytest.mark.parametrize("n,D,nk,nf", [(4, 4, 1, 24), (5, 5, 2, 33), (9, 6, 3, 40), (7, 7, 5, 31), (22, 8, 6, 32),
                                       (32, 9, 9, 24), (10, 10, 4, 65), (28, 10, 17, 47), (32, 10, 26, 24), (9, 5, 3, 33),
                                       (13, 5, 2, 40), (14, 6, 18, 24), (38, 6, 9, 31), (12, 8, 3, 24), (15, 7, 3, 33), (7, 5, 3, 24),
                                       (8, 5, 2, 25), (9, 7, 4, 33), (9, 8, 2, 24), (9, 9, 3, 24)])
def test_tensor_core_block_and_derivative_passes(ctx, orc, n, D, nk, nf):
    """G_loc, GwHF and NumMatrix, and dN/dmu, of the mixed form at 4 <= D <= 10: no ligands up to the 32 poles a k point
    may have, the counts from which each pass is on the tensor cores (0, 2, 4), k counts around the points GwHF's sums
    share and the chunks, frequency counts that leave partial tiles of 32.  Against the FP64 oracle (the mixed tolerance)
    and the GPU's FP64 pass (1e-11: the slices leave less than 2^-41, inversions of matrices of condition < 1e2)."""
    H, S, lat = _random_lattice(n, D, (nk, 1, 1), nf, [n, D, nk])
    for mu in (-0.4, 0.3):
        want = orc.greenftn_w(H, S, mu, 15.0, 1, D)
        f64 = ctx.GreenFtn_w(lat, H, S, mu)
        got = ctx.GreenFtn_w(lat, H, S, mu, mixed=True)
        for g, w, f in zip(got, want, f64):
            assert rel_err(g, w) < TOL_MIXED and rel_err(g, f) < 1e-11
        N, dN = ctx.GiwToNele(lat, H, S, mu, deriv=True)
        g, dg = ctx.GiwToNele(lat, H, S, mu, deriv=True, mixed=True)
        assert abs(g - N) <= 1e-11 * max(1, abs(N)) and abs(dg - dN) <= 1e-10 * max(1, abs(dN))


def test_newton_mu_through_tensor_core_passes(ctx, orc):
    """The mixed Newton mu search on the 28-orbital d+p model (D = 10): its secant passes run on the tensor cores;
    the mu it returns gives the target occupation in the FP64 oracle."""
    wl = models.dp28(k=3, nfreq=64, ntau=256, beta=10.0)
    H = orc.hk(wl.n, wl.rindex, wl.hr, orc.kmesh(*wl.kgrid))
    lat = lib.Lattice(wl.n, wl.nk, wl.nfreq, wl.beta, 1, wl.D)
    mu_n, ne = ctx.GreenFtn_w_adjust_mu(lat, H, wl.sigma, 0.0, 1.0, wl.n_electrons, newton=True, mixed=True)
    assert abs(orc.nele(H, wl.sigma, mu_n, wl.beta, 1, wl.D) - wl.n_electrons) < 1e-9
    mu_c, _ = ctx.GreenFtn_w_adjust_mu(lat, H, wl.sigma, 0.0, 1.0, wl.n_electrons, newton=True, mixed=True,
                                       tensor=False)
    assert abs(mu_n - mu_c) < 1e-9


@pytest.mark.parametrize("case", list(CASES))
def test_mixed_precision_lattice_sum(ctx, orc, case):
    wl = CASES[case]()
    H, lat = _setup(orc, wl)
    gw, gwhf, num = orc.greenftn_w(H, wl.sigma, 0.25, wl.beta, wl.ncl, wl.nh)
    m_gw, m_gwhf, m_num = ctx.GreenFtn_w(lat, H, wl.sigma, 0.25, mixed=True)
    assert rel_err(m_gw, gw) < TOL_MIXED and rel_err(m_gwhf, gwhf) < TOL_MIXED and rel_err(m_num, num) < TOL_MIXED
    N, dN = orc.nele(H, wl.sigma, 0.25, wl.beta, wl.ncl, wl.nh, deriv=True)
    gN, gdN = ctx.GiwToNele(lat, H, wl.sigma, 0.25, deriv=True, mixed=True)
    assert abs(gN - N) < TOL_MIXED * abs(N) and abs(gdN - dN) < 1e-7 * abs(dN)


def test_mixed_precision_newton_mu(ctx, orc):
    wl = CASES["t2g_p"]()
    H, lat = _setup(orc, wl)
    mu_n, ne = ctx.GreenFtn_w_adjust_mu(lat, H, wl.sigma, 0.0, 1.0, 7.3, newton=True, mixed=True)
    assert abs(orc.nele(H, wl.sigma, mu_n, wl.beta, wl.ncl, wl.nh) - 7.3) < 1e-9
    assert ne <= 8


def test_hyb_delta_matches_oracle(ctx, orc):
    wl = CASES["t2g_p"]()
    H, lat = _setup(orc, wl)
    gw, _, _ = orc.greenftn_w(H, wl.sigma, 0.2, wl.beta, wl.ncl, wl.nh)
    himp = H.mean(0)[:3, :3]
    orb = [0, 1, 2]
    d_o = orc.hyb_delta(orb, wl.sigma, gw, himp, 0.2, wl.beta)
    d_g = ctx.Construct_hyb_delta(orb, wl.sigma, gw, 0.2, wl.beta, himp)
    assert rel_err(d_g, d_o) < TOL


@pytest.mark.parametrize("case", ["t2g_p", "dp28", "soc_small"])
@pytest.mark.parametrize("mixed", [False, True])
def test_retarded_gloc_real_axis(ctx, orc, case, mixed):
    """Real-axis lattice sum (retarded_GreenFtn2 over a qs_spectra energy grid) against explicit inversion."""
    if case == "t2g_p":
        wl = models.t2g_p(k=3, nfreq=8, beta=10.0)
    elif case == "dp28":   # D = 10: the packed 10-lane groups
        wl = models.dp28(k=2, nfreq=8, ntau=16, beta=10.0)
    else:
        wl = models.soc56(k=2, nfreq=8, beta=10.0)
    H = orc.hk(wl.n, wl.rindex, wl.hr, orc.kmesh(*wl.kgrid))
    lat = lib.Lattice(wl.n, wl.nk, 8, wl.beta, 1, wl.D)
    nE, e0, de, eta, mu = 40, -4.0, 0.2, 0.05, 0.3
    rng = np.random.default_rng(2)
    A = rng.normal(size=(wl.D, wl.D)) + 1j * rng.normal(size=(wl.D, wl.D))
    Es = e0 + de * np.arange(nE)
    # a causal self-energy on the grid: Hermitian static part - i Gamma(E) (PSD)
    sig = 0.1 * (A + A.conj().T)[None] - 1j * (0.2 + 0.05 * Es[:, None, None] ** 2) * np.eye(wl.D)[None]
    g_o, tr_o = orc.retarded_gloc(H, sig, e0, de, eta, mu, wl.D)
    g, tr = ctx.retarded_GreenFtn(lat, H, sig, e0, de, eta, mu, mixed=mixed)
    tol = 1e-9 if mixed else 1e-10
    assert rel_err(g, g_o) < tol
    assert rel_err(tr, tr_o) < tol


@pytest.mark.parametrize("n,D,nk", [(2, 1, 3), (3, 1, 2), (8, 2, 3), (9, 1, 2), (9, 1, 306), (16, 3, 306), (17, 1, 2), (18, 2, 306),
                                    (19, 2, 5), (31, 8, 2), (32, 10, 3), (33, 1, 2), (63, 2, 1), (64, 3, 2)])
def test_eigensolver_sizes(ctx, orc, n, D, nk):
    """Both decompositions (H + m0: n, H_QQ: n - D) at the edges of their thread groups: odd and even sizes around 8, 16, 32
    and 64, few k points and more than two per SM; with two equal ligand levels and one that nothing couples to.  FP64
    to 1e-11 and the mixed form to the mixed tolerance, as the other passes are held."""
    H, S, lat = _random_lattice(n, D, (nk, 1, 1), 24, [n, D, nk])
    if n - D >= 3:
        H[:, n - 1, :] = H[:, :, n - 1] = 0
        H[:, n - 1, n - 1] = H[:, n - 2, n - 2]
    want = orc.greenftn_w(H, S, 0.2, 15.0, 1, D)
    for mixed, tol in ((False, 1e-11), (True, TOL_MIXED)):
        for g, w in zip(ctx.GreenFtn_w(lat, H, S, 0.2, mixed=mixed), want):
            assert rel_err(g, w) < tol


@pytest.mark.parametrize("dense", ["none", "one frequency", "all"])
@pytest.mark.parametrize("nk,nf,scale", [(1, 24, 1.0), (7, 65, 1.0), (37, 129, 1.0), (5, 24, 1e20)])
def test_nele_two_orbitals_without_ligands(ctx, orc, nk, nf, scale, dense):
    """N(mu) of the 2 x 2 block: the determinant with and without off-diagonal self-energies (in one frequency of a CTA's
    only, too), fractions that run over k points and, with energies of 1e20, past the range of their common denominator.
    FP64 1e-11, double-float 1e-9, as for the other N(mu) passes (double-float: FP32's range, so not at 1e20)."""
    H, S, lat = _random_lattice(2, 2, (nk, 1, 1), nf, [nk, nf])
    if dense != "none":
        f = slice(None) if dense == "all" else slice(nf // 2, nf // 2 + 1)
        S[f, 0, 1] += 0.1 - 0.2j
        S[f, 1, 0] += 0.1 - 0.2j
    for mu in (-0.4, 0.3):
        N = orc.nele(H, S, mu, 15.0, 1, 2)
        N = N[0] if isinstance(N, tuple) else N
        big = lib.Lattice(2, nk, nf, 15.0 / scale, 1, 2)
        assert abs(ctx.GiwToNele(big, H * scale, S * scale, mu * scale) - N) <= 1e-11 * max(1, abs(N))
        if scale == 1.0:
            assert abs(ctx.GiwToNele(lat, H, S, mu, mixed=True) - N) <= 1e-9 * max(1, abs(N))


@pytest.mark.parametrize("n,D,nk,nf", [(4, 4, 3, 33), (8, 4, 2, 65), (5, 5, 3, 24), (18, 7, 5, 33), (8, 8, 2, 31), (9, 8, 7, 32),
                                       (28, 10, 3, 40), (11, 11, 2, 24), (20, 14, 3, 25), (17, 15, 2, 33), (64, 20, 2, 24)])
def test_fp64_passes_by_tiles(ctx, orc, n, D, nk, nf):
    """G_loc, GwHF, NumMatrix and N(mu) in FP64 at the edges of the lane groups (7, 10, 14, 20 orbitals) and of the rule that
    chooses them, with no poles and the most, frequency counts that leave partial CTAs; 1e-11 as for the other FP64 passes."""
    H, S, lat = _random_lattice(n, D, (nk, 1, 1), nf, [n, D, nk, nf])
    for mu in (-0.4, 0.3):
        for g, w in zip(ctx.GreenFtn_w(lat, H, S, mu), orc.greenftn_w(H, S, mu, 15.0, 1, D)):
            assert rel_err(g, w) < 1e-11
        N = orc.nele(H, S, mu, 15.0, 1, D)
        N = N[0] if isinstance(N, tuple) else N
        assert abs(ctx.GiwToNele(lat, H, S, mu) - N) <= 1e-11 * max(1, abs(N))


@pytest.mark.parametrize("n,nk,nf", [(2, 5, 33), (2, 130, 24), (5, 7, 64)])
def test_two_orbital_closed_forms(ctx, orc, n, nk, nf):
    """G_loc, GwHF, NumMatrix, N(mu) and dN/dmu of 2 x 2 blocks with a dense self-energy whose determinant has its larger
    product off the diagonal (the pivot's place), with and without ligands; the bounds of the other sizes."""
    H, S, lat = _random_lattice(n, 2, (nk, 1, 1), nf, [n, nk])
    H[:, 0, 1] += 3.0
    H[:, 1, 0] += 3.0
    for mu in (-0.4, 0.3):
        want = orc.greenftn_w(H, S, mu, 15.0, 1, 2)
        N, dN = orc.nele(H, S, mu, 15.0, 1, 2, deriv=True)
        for mixed, tol in ((False, 1e-11), (True, TOL_MIXED)):
            for g, w in zip(ctx.GreenFtn_w(lat, H, S, mu, mixed=mixed), want):
                assert rel_err(g, w) < tol
            g, dg = ctx.GiwToNele(lat, H, S, mu, deriv=True, mixed=mixed)
            assert abs(g - N) <= tol * max(1, abs(N)) and abs(dg - dN) <= 10 * tol * max(1, abs(dN))


@pytest.mark.parametrize("D", [1, 4, 6])
def test_k_sum_keeps_its_digits(ctx, D):
    """20,000 k points and 32 frequencies: the sum is split into some thousand chunks, which one running sum would add up with
    an error of 12 u (u = 2^-53; u/sqrt(3) per addition, of a partial sum of 0.58 of the total, sqrt(1,216) of them).  The
    blocks of 64 make it 1.5 u; the bound is three times that.  Diagonal H, so that the sums are of scalars (long double)."""
    rng = np.random.default_rng(D)
    nk, nf, beta, mu = 20000, 16, 20.0, 0.2
    e = rng.normal(size=(nk, D))
    H = np.zeros((nk, D, D), complex)
    H[:, range(D), range(D)] = e
    w = np.pi * (2 * np.arange(nf) + 1) / beta
    S = (-0.5j / (w + 1.0))[:, None, None] * np.eye(D)
    G = ctx.GreenFtn_w(lib.Lattice(D, nk, nf, beta, 1, D), H, S, mu)[0]
    z = (np.longdouble(mu) - e)[:, :, None] + np.clongdouble(1j) * (w + 0.5 / (w + 1.0)).astype(np.longdouble)
    exact = (1 / z).sum(0) / nk                                        # [D][nf]
    err = np.array([G[:, a, a] - exact[a] for a in range(D)])
    assert np.sqrt((abs(err) ** 2).sum() / (abs(exact) ** 2).sum()) < 4.5 * 2.0 ** -53


def test_mixed_passes_without_room_for_operand_images(ctx):
    """24,000 k points whose operand images (2.1 GB for G_loc, 1.0 for N(mu)) do not fit in what is left of the device: the
    passes run without them, as with tensor=False, and the next call with room takes the tensor cores again."""
    import torch
    n, D, nk, nf = 14, 10, 24000, 8
    g = torch.Generator(device="cuda").manual_seed(5)
    A = torch.view_as_complex(torch.randn(nk, n, n, 2, dtype=torch.float64, device="cuda", generator=g))
    H = (A + A.conj().transpose(1, 2)) / 4
    S = torch.eye(D, dtype=torch.complex128, device="cuda").repeat(nf, 1, 1) * (-0.2j)
    lat = lib.Lattice(n, nk, nf, 10.0, 1, D)
    want = [ctx.GiwToNele(lat, H, S, 0.3, mixed=True, tensor=False), ctx.GiwToNele(lat, H, S, 0.3, deriv=True, mixed=True, tensor=False)]
    full = ctx.GreenFtn_w(lat, H, S, 0.3)[0].cpu()
    c = lib.Context(0)
    hog = None
    try:
        c.GiwToNele(lat, H, S, 0.3, mixed=True, tensor=False)      # what every pass needs is there
        c.GreenFtn_w(lat, H, S, 0.3)
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        hog = torch.empty(free - (900 << 20), dtype=torch.uint8, device="cuda")
        got = [c.GiwToNele(lat, H, S, 0.3, mixed=True), c.GiwToNele(lat, H, S, 0.3, deriv=True, mixed=True)]
        G = c.GreenFtn_w(lat, H, S, 0.3, mixed=True)[0].cpu()
        assert got == want
        assert float((G - full).abs().max() / full.abs().max()) < TOL_MIXED
        n0 = c.launches()
        c.GreenFtn_w(lat, H, S, 0.3, mixed=True)
        without = c.launches() - n0
        del hog
        hog = None
        torch.cuda.empty_cache()
        n0 = c.launches()
        G = c.GreenFtn_w(lat, H, S, 0.3, mixed=True)[0].cpu()
        assert c.launches() - n0 != without
        assert float((G - full).abs().max() / full.abs().max()) < TOL_MIXED
    finally:
        del hog
        torch.cuda.empty_cache()
        c.close()


def test_tensor_switch_of_the_lattice_sum(ctx, orc):
    """tensor=False keeps G_loc and GwHF of a 10-orbital block off the tensor cores, alone and in a batch (fewer launches: no
    operand images), with the oracle's values either way."""
    import torch
    wl = models.dp28(k=2, nfreq=24, ntau=16, beta=20.0)
    H, lat = _setup(orc, wl)
    ref = orc.greenftn_w(H, wl.sigma, 0.2, wl.beta, wl.ncl, wl.nh)
    n, cm = [], lambda x: torch.from_numpy(np.ascontiguousarray(x.transpose(0, 2, 1))).cuda()
    for tensor in (True, False):
        n0 = ctx.launches()
        G, G0, N = ctx.GreenFtn_w(lat, H, wl.sigma, 0.2, mixed=True, tensor=tensor)
        n.append(ctx.launches() - n0)
        for x, y in zip((G, G0, N), ref):
            assert rel_err(x, y) < TOL_MIXED
        out = [torch.zeros((wl.nfreq, wl.D, wl.D), dtype=torch.complex128, device="cuda") for _ in range(2)]
        num = torch.zeros((wl.D, wl.D), dtype=torch.complex128, device="cuda")
        n0 = ctx.launches()
        ctx.GreenFtn_w_batched([lat], [cm(H)], [cm(wl.sigma)], [0.2], out[:1], out[1:], [num], mixed=True, tensor=tensor)
        assert ctx.launches() - n0 == n[-1]
        assert rel_err(out[0].transpose(1, 2).cpu().numpy(), G) == 0.0
    assert n[1] < n[0]


@pytest.mark.parametrize("n,nk,nf", [(15, 5, 33), (16, 1, 24), (16, 7, 31), (11, 4, 40), (12, 3, 25), (36, 9, 48), (32, 20, 64),
                                     (37, 2, 24)])
def test_nele_of_four_orbitals_with_many_ligands(ctx, n, nk, nf):
    """N(mu) and dN/dmu of 4 x 4 blocks below, at and above the pole counts (12, 8; 32 the most) from which their pole sums are on
    the tensor cores, partial tiles of 32 frequencies and single k points among them: the mixed form against FP64 within
    the slices' 2^-41 of sums over matrices of condition < 1e2, and against its form on the CUDA cores."""
    H, S, lat = _random_lattice(n, 4, (nk, 1, 1), nf, [n, 4, nk])
    for mu in (-0.4, 0.3):
        N, dN = ctx.GiwToNele(lat, H, S, mu, deriv=True)
        for tensor in (True, False):
            g = ctx.GiwToNele(lat, H, S, mu, mixed=True, tensor=tensor)
            assert abs(g - N) <= 1e-11 * max(1, abs(N))
            g, dg = ctx.GiwToNele(lat, H, S, mu, deriv=True, mixed=True, tensor=tensor)
            assert abs(g - N) <= 1e-11 * max(1, abs(N)) and abs(dg - dN) <= 1e-10 * max(1, abs(dN))


@pytest.mark.parametrize("n,D", [(16, 4), (10, 6), (14, 10)])
def test_units_of_energy(ctx, n, D):
    """All energies times 2^40 and beta by 2^-40: the same numbers in other units, dN/dmu smaller by 2^40.  The pole sums' rows of
    w^3 are 1e-36 and less then, their low halves beyond FP32: digits go (2^-20 of dN/dmu are left), the number does not."""
    H, S, lat = _random_lattice(n, D, (5, 1, 1), 40, [n, D])
    N, dN = ctx.GiwToNele(lat, H, S, 0.3, deriv=True, mixed=True)
    big = lib.Lattice(n, lat.nk, lat.nfreq, lat.beta / 2.0 ** 40, 1, D)
    M, dM = ctx.GiwToNele(big, H * 2.0 ** 40, S * 2.0 ** 40, 0.3 * 2.0 ** 40, deriv=True, mixed=True)
    assert abs(M - N) <= 1e-11 * abs(N) and abs(dM * 2.0 ** 40 - dN) <= 2.0 ** -20 * abs(dN)
