"""Inputs that are not finite: every lattice call refuses them with an error status, and the context goes on."""
import numpy as np
import pytest

from conftest import rel_err
from dmftpack_gb300 import lib

pytestmark = pytest.mark.gpu


def _problem(n, D, nk=6, nf=32, seed=3):
    rng = np.random.default_rng([seed, n, D])
    H = rng.normal(size=(nk, n, n)) + 1j * rng.normal(size=(nk, n, n))
    w = np.pi * (2 * np.arange(nf) + 1) / 20.0
    S = -1j * 0.5 / (w[:, None, None] + 1.0) * np.eye(D)
    return lib.Lattice(n, nk, nf, 20.0, 1, D), (H + H.conj().transpose(0, 2, 1)) / 2, S


@pytest.mark.parametrize("n,D", [(2, 2), (5, 3), (12, 5), (20, 4), (28, 10), (40, 12)])
@pytest.mark.parametrize("mixed", [False, True])
def test_nan_is_refused(ctx, n, D, mixed):
    """NaN in one k point's H, or in Sigma: the eigenvalues of whole k points are NaN then, and their order still has to
    address eigenvectors (one warp and four warps per matrix, both arithmetics)."""
    lat, H, S = _problem(n, D)
    good = ctx.GreenFtn_w(lat, H, S, 0.1, mixed=mixed)[0]
    bad = H.copy()
    bad[2, n - 1, n - 1] = bad[4, 0, 0] = np.nan
    for h, s in ((bad, S), (H, np.where(np.arange(len(S))[:, None, None] == len(S) - 1, np.nan, S))):
        with pytest.raises(lib.DmftGpuError):
            ctx.GreenFtn_w(lat, h, s, 0.1, mixed=mixed)
        with pytest.raises(lib.DmftGpuError):
            ctx.GiwToNele(lat, h, s, 0.1, mixed=mixed)
        with pytest.raises(lib.DmftGpuError):
            ctx.densityMatDFT(lat, h, s, 0.1, mixed=mixed)
        with pytest.raises(lib.DmftGpuError):
            ctx.GreenFtn_w_vjp(lat, h, s, 0.1, S)
    assert rel_err(ctx.GreenFtn_w(lat, H, S, 0.1, mixed=mixed)[0], good) == 0.0


@pytest.mark.parametrize("n,D", [(1, 1), (5, 3), (12, 8), (20, 20)])
def test_derivatives_refuse_an_infinite_self_energy(ctx, n, D):
    """An infinite last pivot: |pivot|^2 is not zero, but there is no inverse."""
    lat, H, S = _problem(n, D)
    bad = S.copy()
    bad[3, D - 1, D - 1] = np.inf
    good = ctx.GreenFtn_w_jvp(lat, H, S, 0.1, S, 0.2)
    with pytest.raises(lib.DmftGpuError):
        ctx.GreenFtn_w_jvp(lat, H, bad, 0.1, S, 0.2)
    with pytest.raises(lib.DmftGpuError):
        ctx.GreenFtn_w_vjp(lat, H, bad, 0.1, S)
    assert rel_err(ctx.GreenFtn_w_jvp(lat, H, S, 0.1, S, 0.2), good) == 0.0
