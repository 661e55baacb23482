"""The calls this library is timed on: the lattice sum, the chemical-potential search, H(k), the derivatives, the
per-k density matrix, the batched pass, the SC2PT impurity solver and a whole DMFT iteration, over the sizes of the
benchmark configurations (dmftpack_gb300/models.py), the reference's example input and ragged ones between them.

Inputs are built here from the seed alone with plain numpy / torch (hoppings t(R), H(k), Sigma), so they do not depend
on the library; `exact` evaluates the defining formulas in 64 bits with full or block inversions, without it.
"""
import math

import numpy as np
import torch

from dmftpack_gb300 import lib, models

PI = math.pi
_ctx = None


def context():
    """The one library handle a program keeps."""
    global _ctx
    if _ctx is None:
        _ctx = lib.Context(0)
    return _ctx


# ------------------------------------------------------------------------------------------------------------------
# cases
# ------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the reference's example input (22 x 22 x 1 k, N_MATSUBARA = 400): the smallest call, host arrays as a C++
        # program passes them
        dict(name="gloc_example", kind="gloc", model="hubbard", n=2, D=2, kx=22, ky=22, kz=1, nfreq=400, beta=40.0,
             mixed=False, host=True),
        # the headline lattice sum of the t2g + p model at its full size
        dict(name="gloc_t2gp", kind="gloc", model="dp", n=12, D=3, kx=24, ky=24, kz=24, nfreq=4096, beta=40.0,
             mixed=True, host=False),
        # the same model in plain FP64 on an ordinary odd mesh
        dict(name="gloc_t2gp_f64", kind="gloc", model="dp", n=12, D=3, kx=13, ky=13, kz=13, nfreq=1000, beta=40.0,
             mixed=False, host=False),
        # the lattice sum of the 28-orbital d + p model (ten correlated spin-orbitals)
        dict(name="gloc_dp28", kind="gloc", model="dp", n=28, D=10, kx=10, ky=10, kz=10, nfreq=2048, beta=40.0,
             mixed=True, host=False),
        # the reference's bisection for mu on the square-lattice Hubbard configuration, FP64
        dict(name="mu_hubbard_bisect", kind="mu", model="hubbard", n=2, D=2, kx=64, ky=64, kz=1, nfreq=2048,
             beta=50.0, mixed=False, newton=False),
        # the Newton search for mu of the d + p model
        dict(name="mu_dp28_newton", kind="mu", model="dp", n=28, D=10, kx=8, ky=8, kz=8, nfreq=2048, beta=40.0,
             mixed=True, newton=True),
        # H(k) from the 729-vector hopping table of the d + p model
        dict(name="hk_dp28", kind="hk", n=28, rmax=4, kx=20, ky=20, kz=20, mixed=True),
        # tangent, then adjoint of the lattice sum on the 56-orbital spin-orbit model with a dense 20 x 20 Sigma: one
        # Gauss-Newton product J^H J v of a fit to G_loc
        dict(name="derivs_soc56", kind="derivs", model="soc", n=56, D=20, kx=5, ky=5, kz=5, nfreq=512, beta=30.0),
        # the per-k density matrix handed back to the DFT code
        dict(name="density_dp28", kind="density", model="dp", n=28, D=10, kx=6, ky=6, kz=6, nfreq=1024, beta=40.0,
             mixed=True),
        # a batch of independent lattice problems of ragged sizes
        dict(name="batch_ragged", kind="batch", nprob=12, kmax=12, nfmax=1024, mixed=True),
        # the SC2PT solver of ten spin-orbitals, some loops of a run
        dict(name="scgf2_d10", kind="scgf2", d=10, nfreq=4096, ntau=8192, beta=40.0, loops=12, mixed=True),
        # one whole DMFT iteration of the square-lattice Hubbard configuration with IPT
        dict(name="dmft_hubbard_ipt", kind="dmft", kx=64, ky=64, nfreq=2048, ntau=8192, beta=50.0, U=2.0, mixed=True,
             newton=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, most):
    """kx x ky x kz <= most, sides not all equal."""
    side = max(1, int(most ** (1 / 3)))
    k = [max(1, rng.randint(max(1, side - 3), side)) for _ in range(3)]
    return k


def draw(rng):
    kind = rng.choice(["gloc", "gloc", "gloc", "mu", "hk", "derivs", "density", "batch", "scgf2", "dmft"])
    if kind in ("gloc", "mu"):
        mixed = rng.random() < 0.65
        D = rng.randint(1, 10)
        n = min(32, D + rng.randint(0, 22)) if rng.random() < 0.8 else D
        nf = _log_int(rng, 64, 4096)
        # points so that one pass stays within the listed ones' time
        cost = ((n - D) * D * D + 2 * D ** 3 + 40) * (1 if mixed else 6)
        most = (1.2e10 if kind == "gloc" else 4e9 if mixed else 1.2e9) / cost / (2 * nf)
        # (the mu search on meshes that are not a handful of levels)
        least = 8 if kind == "gloc" else 64
        most = max(least, min(_log_int(rng, least, 8000), int(most)))
        kx, ky, kz = _mesh(rng, most)
        c = dict(kind=kind, model="dp", n=n, D=D, kx=kx, ky=ky, kz=kz, nfreq=nf,
                 beta=round(rng.uniform(10, 100 if kind == "gloc" else 50), 3), mixed=mixed)
        return dict(c, host=False) if kind == "gloc" else dict(c, newton=mixed)
    if kind == "hk":
        kx, ky, kz = _mesh(rng, _log_int(rng, 64, 8000))
        return dict(kind=kind, n=rng.randint(2, 28), rmax=rng.randint(1, 4), kx=kx, ky=ky, kz=kz,
                    mixed=rng.random() < 0.7)
    if kind == "derivs":
        D = rng.randint(2, 20)
        n = min(56, D + rng.randint(0, 36))
        nf = _log_int(rng, 32, 1024)
        most = 1.5e9 / ((n - D) * D * D + 4 * D ** 3 + 100) / nf
        kx, ky, kz = _mesh(rng, max(8, min(1000, int(most))))
        return dict(kind=kind, model="dp", n=n, D=D, kx=kx, ky=ky, kz=kz, nfreq=nf, beta=round(rng.uniform(10, 60), 3))
    if kind == "density":
        D = rng.randint(2, 10)
        n = min(28, D + rng.randint(1, 18))
        nf = _log_int(rng, 64, 1024)
        mixed = rng.random() < 0.7
        most = 2.5e9 / (n ** 3 * (1 if mixed else 4)) / (2 * nf)
        kx, ky, kz = _mesh(rng, max(8, min(1000, int(most))))
        return dict(kind=kind, model="dp", n=n, D=D, kx=kx, ky=ky, kz=kz, nfreq=nf, beta=round(rng.uniform(10, 60), 3),
                    mixed=mixed)
    if kind == "batch":
        return dict(kind=kind, nprob=rng.randint(2, 12), kmax=rng.randint(5, 12), nfmax=_log_int(rng, 256, 1024),
                    mixed=rng.random() < 0.8)
    if kind == "scgf2":
        d = 2 * rng.randint(1, 5)
        nf = rng.choice([512, 800, 1024, 2000, 2048, 4096])
        # powers of two take the FFT path, others the direct sums (as the example's N_TAU = 2400 does)
        ntau = 2 * nf if nf & (nf - 1) == 0 else min(2 * nf, 2000)
        return dict(kind=kind, d=d, nfreq=nf, ntau=ntau, beta=round(rng.uniform(20, 60), 3), loops=rng.randint(11, 13),
                    mixed=rng.random() < 0.7)
    nf = rng.choice([512, 1024, 2048])
    return dict(kind=kind, kx=rng.randint(12, 64), ky=rng.randint(12, 64), nfreq=nf, ntau=4 * nf,
                beta=round(rng.uniform(20, 50), 3), U=round(rng.uniform(1.0, 3.0), 3), mixed=rng.random() < 0.7,
                newton=True)


# ------------------------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------------------------
def _rvecs(rmax):
    r = np.arange(-rmax, rmax + 1)
    return np.stack(np.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 3)


def _random_hoppings(rng, n, rmax, scale, onsite):
    """t(R) ~ scale N(0, 1)/|R|^2 complex with t(-R) = t(R)^H on the cube |R_i| <= rmax."""
    R = _rvecs(rmax)
    nR = len(R)
    r2 = np.maximum(1, (R ** 2).sum(1))
    T = (rng.normal(size=(nR, n, n)) + 1j * rng.normal(size=(nR, n, n))) * (scale / np.sqrt(2) / r2)[:, None, None]
    half = nR // 2  # R[nR - 1 - i] = -R[i]
    T[nR - 1:half:-1] = T[:half].conj().transpose(0, 2, 1)
    T[half] = (T[half] + T[half].conj().T) / 2 + np.diag(onsite)
    return R, T


def _ls_d():
    m = np.arange(-2, 3)
    lz = np.diag(m).astype(complex)
    lp = np.zeros((5, 5), complex)
    for i in range(4):
        lp[i + 1, i] = math.sqrt(6 - m[i] * (m[i] + 1))
    sz, sp = np.diag([0.5, -0.5]).astype(complex), np.array([[0, 1], [0, 0]], complex)
    return np.kron(lz, sz) + 0.5 * (np.kron(lp, sp.T) + np.kron(lp.T, sp))


def _model(c, seed):
    """(R[nR, 3], T[nR, n, n]) of a case's model."""
    rng = np.random.default_rng([int(seed), 1])
    model, n, D = c["model"], c["n"], c["D"]
    if model == "hubbard":
        t, tp = 1.0 + 0.05 * rng.uniform(), -0.25 + 0.05 * rng.uniform()
        R = np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [1, 1, 0], [1, -1, 0], [-1, 1, 0], [-1, -1, 0]])
        return R, np.array([-t] * 4 + [-tp] * 4)[:, None, None] * np.eye(2)[None].astype(complex)
    if model == "soc":
        norb = n // 2
        onsite = np.array([0.0] * (D // 2) + [-3.0] * (norb - D // 2))
        R, t = _random_hoppings(rng, norb, 3, 0.5, onsite)
        T = np.kron(t, np.eye(2))
        for site in range(D // 10):
            T[len(R) // 2, 10 * site:10 * site + 10, 10 * site:10 * site + 10] += 0.1 * _ls_d()
        return R, T
    onsite = np.array([0.0] * D + [-3.0] * (n - D))
    return _random_hoppings(rng, n, 1 if n > 28 else 2, 1.0 if n <= 16 else 0.5, onsite)


def _hk(R, T, kx, ky, kz, dev):
    """H(k) = sum_R T(R) e^{-i k.aR}, k.a = -pi + pi/N + 2 pi i/N on each axis, the first axis fastest."""
    nk = kx * ky * kz
    i = torch.arange(nk, device=dev)
    ix, iy, iz = i % kx, (i // kx) % ky, i // (kx * ky)
    ka = torch.stack([-PI + PI / m + j.double() * (2 * PI / m) for j, m in ((ix, kx), (iy, ky), (iz, kz))], 1)
    R = torch.as_tensor(np.ascontiguousarray(R), dtype=torch.float64, device=dev)
    n = T.shape[1]
    Tt = torch.as_tensor(np.ascontiguousarray(T), dtype=torch.complex128, device=dev).reshape(len(T), n * n)
    out = torch.empty(nk, n, n, dtype=torch.complex128, device=dev)
    for a in range(0, nk, 4096):
        ang = ka[a:a + 4096] @ R.T
        out[a:a + 4096] = (torch.polar(torch.ones_like(ang), -ang) @ Tt).reshape(-1, n, n)
    return out


def _cm(x):
    """The layout Construct_Hk returns: logical (count, i, j), stored column-major per matrix."""
    return x.transpose(-1, -2).contiguous().transpose(-1, -2)


def _wn(nf, beta, dev="cpu"):
    return PI * (2 * torch.arange(nf, dtype=torch.float64, device=dev) + 1) / beta


def _sigma(c, seed, dev):
    """Self-energy of the workloads: diagonal, Im Sigma = -g/(w + h) (dense M0 + M1/(iw) for the spin-orbit model)."""
    rng = np.random.default_rng([int(seed), 2])
    D, w = c["D"], _wn(c["nfreq"], c["beta"], dev)
    if c["model"] == "soc":
        A = rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D))
        B = rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D))
        M0, M1 = (torch.as_tensor(m, device=dev) for m in (0.1 * (A + A.conj().T), 0.1 * B @ B.conj().T / D))
        return M0[None] + M1[None] / (1j * w[:, None, None])
    g = torch.as_tensor(rng.uniform(0.4, 0.6, D), device=dev)
    h = torch.as_tensor(rng.uniform(0.8, 1.2, D), device=dev)
    if c["model"] == "hubbard":
        g, h = g[:1].expand(D), h[:1].expand(D)
    return torch.diag_embed(-1j * g / (w[:, None] + h))


def _fill(c):
    """Electron count the mu search aims at."""
    return 1.0 if c["model"] == "hubbard" else 0.6137 * c["n"]


def _batch(c, seed):
    """Ragged problems: dimension from {1, 3, 5, 10, 14, 28} and odd ones between, k^3 meshes, N_freq."""
    shape = np.random.default_rng([c["nprob"], c["kmax"], c["nfmax"]])
    dims = [1, 3, 5, 10, 14, 28, 7, 2]
    out = []
    for i in range(c["nprob"]):
        n = dims[i % len(dims)]
        k = int(shape.integers(4, c["kmax"] + 1)) if n < 28 else min(6, c["kmax"])
        out.append(dict(kind="gloc", model="dp", n=n, D=min(n, 10), kx=k, ky=k, kz=max(1, k - 1),
                        nfreq=int(shape.integers(128, c["nfmax"] + 1)), beta=float(shape.uniform(10, 100)),
                        mixed=c["mixed"], host=False, seed=int(seed) * 64 + i))
    return out


def _impurity(c, seed):
    """H_imp, Delta(iw) and a starting G_imp of a d-orbital impurity: dense random levels and eight bath poles."""
    rng = np.random.default_rng([int(seed), 3])
    d, nf = c["d"], c["nfreq"]
    A = rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d))
    himp = 0.3 * (A + A.conj().T) / 2
    iw = 1j * _wn(nf, c["beta"]).numpy()[:, None, None]
    delta = np.zeros((nf, d, d), complex)
    for e in rng.uniform(-3, 3, size=8):
        v = 0.4 * (rng.normal(size=d) + 1j * rng.normal(size=d))
        delta += np.outer(v, v.conj())[None] / (iw - e)
    mu = 0.5
    return himp, delta, np.linalg.inv((iw + mu) * np.eye(d)[None] - himp[None] - delta), mu


def prepare(case, seed):
    c, dev = case, torch.device("cuda", 0)
    kind = c["kind"]
    s = dict(c, ctx=context())
    if kind == "batch":
        s["lats"], s["H"], s["S"], s["mu"], s["out"] = [], [], [], [], []
        for p in _batch(c, seed):
            q = prepare({k: v for k, v in p.items() if k != "seed"}, p["seed"])
            n, D, nf = p["n"], p["D"], p["nfreq"]
            s["lats"].append(q["lat"])
            s["H"].append(q["H"].transpose(-1, -2).contiguous())
            s["S"].append(q["S"].transpose(-1, -2).contiguous())
            s["mu"].append(q["mu"])
            s["out"].append([torch.zeros(nf, D, D, dtype=torch.complex128, device=dev) for _ in range(2)] +
                            [torch.zeros(D, D, dtype=torch.complex128, device=dev)])
        return s
    if kind == "scgf2":
        # a handle of its own: the solver's mixing control remembers the previous call's residual
        s["ctx"] = lib.Context(0)
        himp, delta, g0, s["mu"] = _impurity(c, seed)
        s["himp"], s["delta"], s["g0"] = (torch.as_tensor(x, device=dev) for x in (himp, delta, g0))
        s["uidx"], s["ut"] = models.gen_Uijkl(c["d"], 4.0, 2.6, 0.7)
        return s
    if kind == "hk":
        rng = np.random.default_rng([int(seed), 1])
        n = c["n"]
        R, T = _random_hoppings(rng, n, c["rmax"], 0.5, np.linspace(-3, 0, n))
        e = np.stack(np.meshgrid(np.arange(n), np.arange(n), indexing="ij"), -1).reshape(-1, 2)
        s["rindex"] = np.concatenate([np.repeat(R, n * n, 0), np.tile(e, (len(R), 1))], 1).astype(np.int32)
        s["hr"] = np.ascontiguousarray(T.reshape(-1))
        return s
    if kind == "dmft":
        c = dict(c, model="hubbard", n=2, D=2, kz=1)
    R, T = _model(c, seed)
    H = _hk(R, T, c["kx"], c["ky"], c["kz"], dev)
    s["lat"] = lib.Lattice(c["n"], H.shape[0], c["nfreq"], c["beta"], 1, c["D"])
    rng = np.random.default_rng([int(seed), 4])
    if kind == "dmft":
        # the state after a first TightBinding call with the seeded Sigma = U^2/(4 iw)
        w = _wn(c["nfreq"], c["beta"], dev)
        eye = torch.eye(2, dtype=torch.complex128, device=dev)
        sig = (c["U"] ** 2 / 4 * (1 + 0.1 * rng.uniform())) / (1j * w)
        mu = -0.4 + 0.1 * rng.uniform()
        e = H[:, 0, 0].real
        g = torch.cat([(1 / (1j * x[:, None] + mu - y[:, None] - e[None])).mean(1)
                       for x, y in zip(w.split(256), sig.split(256))])
        himp = H[:, 0, 0].mean()
        s["H_cm"] = H.transpose(-1, -2).contiguous()
        s["state"] = [(x[:, None, None] * eye).contiguous() for x in (sig, 1j * w + mu - himp - sig - 1 / g, g)]
        s["num"] = (0.5 + 0.02 * rng.uniform()) * eye
        s["mu"] = mu
        uidx, ut = models.gen_Uijkl(2, c["U"], c["U"], 0.0, density_density=True)
        s["params"] = dict(ntau=c["ntau"], n_electrons=1.0, U=c["U"], Uprime=c["U"], J=0.0, mixing=0.5, magnetism=0,
                           dctype=1, nominal_charge=1.0, uidx=uidx, ut=ut)
        return s
    s["H"], s["S"] = _cm(H), _sigma(c, seed, dev)
    s["mu"] = float(rng.uniform(-0.5, 0.5))
    if c.get("host"):
        s["H"], s["S"] = s["H"].cpu().numpy(), s["S"].cpu().numpy()
    if kind == "derivs":
        D, nf = c["D"], c["nfreq"]
        sd = rng.normal(size=(nf, D, D)) + 1j * rng.normal(size=(nf, D, D))
        s["Sdot"], s["mudot"] = torch.as_tensor(sd, device=dev), float(rng.uniform(0.1, 1.0))
    return s


# ------------------------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------------------------
def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "gloc":
        return ctx.GreenFtn_w(s["lat"], s["H"], s["S"], s["mu"], mixed=s["mixed"])
    if kind == "mu":
        got = ctx.GreenFtn_w_adjust_mu(s["lat"], s["H"], s["S"], s["mu"], 1.0, _fill(s), newton=s["newton"],
                                       mixed=s["mixed"])
        # the bisection's number of passes is the reference's; the Newton search's is not part of its result
        return got[:1] if s["newton"] else got
    if kind == "hk":
        return ctx.Construct_Hk(s["n"], s["rindex"], s["hr"], (s["kx"], s["ky"], s["kz"]),
                                device_out=torch.device("cuda", 0), mixed=s["mixed"])
    if kind == "derivs":
        gd = ctx.GreenFtn_w_jvp(s["lat"], s["H"], s["S"], s["mu"], s["Sdot"], s["mudot"])
        sb, mb = ctx.GreenFtn_w_vjp(s["lat"], s["H"], s["S"], s["mu"], gd)
        return gd, sb, mb
    if kind == "density":
        return ctx.densityMatDFT(s["lat"], s["H"], s["S"], s["mu"], mixed=s["mixed"])
    if kind == "batch":
        gw, g0, nm = ([o[i] for o in s["out"]] for i in range(3))
        ctx.GreenFtn_w_batched(s["lats"], s["H"], s["S"], s["mu"], gw, g0, nm, mixed=s["mixed"])
        return [[x.transpose(-1, -2) for x in o] for o in s["out"]]
    if kind == "scgf2":
        se, g, loops = ctx.SCGF2(s["himp"], s["delta"], s["g0"], s["uidx"], s["ut"], s["mu"], s["beta"], s["ntau"],
                                 0.5, max_iter=s["loops"], mixed=s["mixed"])
        return se, g, loops
    se, we, gl = (x.clone() for x in s["state"])
    nm = s["num"].clone()
    mu, gi, res = ctx.DMFT_iteration(s["lat"], s["H_cm"], s["params"], 1, se, we, nm, gl, s["mu"], mixed=s["mixed"],
                                     newton=s["newton"])
    return dict(mu=mu, gimp=gi, resid=res, selfe=se, weiss=we, nummat=nm, gloc=gl)


# ------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------------------
def work(c):
    kind = c["kind"]
    if kind == "batch":
        w = [work(p) for p in _batch(c, 0)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    if kind == "scgf2":
        d, nu = c["d"], len(models.gen_Uijkl(c["d"], 4.0, 2.6, 0.7)[1])
        per = (c["ntau"] + 1) * 52.0 * nu * nu / d + c["nfreq"] * 8.0 * d ** 3
        per += 2 * d * d * 5.0 * c["ntau"] * math.log2(c["ntau"])
        return {"bytes": 16.0 * d * d * 5 * c["nfreq"], "flops": c["loops"] * per}
    if kind == "dmft":
        c = dict(c, n=2, D=2, kz=1)
    nk, n = c["kx"] * c["ky"] * c["kz"], c["n"]
    if kind == "hk":
        nR = (2 * c["rmax"] + 1) ** 3
        return {"bytes": 16.0 * n * n * (nk + nR), "flops": 8.0 * nk * nR * n * n}
    D, nf = c["D"], c["nfreq"]
    m, nbytes = n - D, 16.0 * nk * n * n + 16.0 * nf * D * D
    if kind == "gloc":
        return {"bytes": nbytes + 32.0 * nf * D * D, "flops": nk * 2.0 * nf * (8.0 * m * D * D + 16.0 * D ** 3)}
    if kind == "mu":
        return {"bytes": nbytes, "flops": (6 if c["newton"] else 20) * nk * 2.0 * nf * 8.0 * (m * D * D + D ** 3)}
    if kind == "derivs":
        return {"bytes": nbytes + 48.0 * nf * D * D,
                "flops": nk * 1.0 * nf * 8.0 * (2 * (2 * m * D * D + D ** 3) + 4 * D ** 3)}
    if kind == "density":
        return {"bytes": nbytes + 16.0 * nk * n * n,
                "flops": nk * 2.0 * nf * 8.0 * (3 * m * D * D + D ** 3 + D * m * m)}
    return {"bytes": nbytes + 80.0 * nf * 4, "flops": 8 * nk * 2.0 * nf * 8.0 * D ** 3}


# ------------------------------------------------------------------------------------------------------------------
# the same quantities in 64 bits, from their definitions
# ------------------------------------------------------------------------------------------------------------------
def _moments(S, beta):
    """getAsymto_moments of S[nf, D, D]: least-squares fits m0 + m1/iw + m2/(iw)^2 + m3/(iw)^3 on the windows
    [w, nf), averaged over 2 nf/20 + 1 consecutive windows; per moment the averaging range of least variance among those
    whose averaged moments describe a positive tail."""
    S = S.cpu().numpy()
    nf, D = S.shape[:2]
    w = PI * (2 * np.arange(nf) + 1) / beta
    Sh = S.conj().transpose(0, 2, 1)
    re, im = (S + Sh) / 2, (S - Sh) / 2j
    suf = lambda x: np.cumsum(x[::-1], 0)[::-1]
    z = w[:, None, None]
    s0, s2, s1, s3 = suf(re), suf(-re / z ** 2), suf(-im / z), suf(im / z ** 3)
    one, a, b = suf(np.ones(nf)), suf(-1 / w ** 2), suf(1 / w ** 4)
    p, q, r = suf(1 / w ** 2), suf(-1 / w ** 4), suf(1 / w ** 6)
    nR = nf - 3
    x = lambda v: v[:nR, None, None]
    d02, d13 = x(one * b - a * a), x(p * r - q * q)
    mt = np.stack([(x(b) * s0[:nR] - x(a) * s2[:nR]) / d02, (x(r) * s1[:nR] - x(q) * s3[:nR]) / d13,
                   (x(one) * s2[:nR] - x(a) * s0[:nR]) / d02, (x(p) * s3[:nR] - x(q) * s1[:nR]) / d13])
    nv = max(1, nf // 20)
    L, C = 2 * nv + 1, nR - 2 * nv
    win = np.lib.stride_tricks.sliding_window_view
    avg = win(mt, L, axis=1).mean(-1)[:, :C]
    var = win(np.trace(mt, axis1=2, axis2=3).real, L, axis=1).std(-1)[:, :C]
    m1, m2, m3 = avg[1], avg[2], avg[3]
    ev, U = np.linalg.eigh(m1)
    ok = ev[:, 0] > 0
    vi = (U / np.sqrt(np.where(ev > 0, ev, 1.0))[:, None, :]) @ U.conj().transpose(0, 2, 1)
    y = vi @ m2 @ vi
    ok &= np.linalg.eigvalsh(vi @ m3 @ vi - y @ y)[:, 0] > 0
    out = []
    for i in range(4):
        good = np.where(ok & (var[i] < var[i, -1]), var[i], np.inf)
        k = int(np.argmin(good)) if np.isfinite(good).any() else C - 1
        mm = mt[i, k:k + L].mean(0)
        out.append((mm + mm.conj().T) / 2)
    return out


def _tail(S, beta, mom):
    """Sigma on 2 nf Matsubara points: the data, then its moment expansion."""
    nf = S.shape[0]
    w = _wn(2 * nf, beta, S.device)[nf:, None, None]
    m = [torch.as_tensor(x, device=S.device) for x in mom]
    return torch.cat([S, m[0] + m[1] / (1j * w) - m[2] / w ** 2 + 1j * m[3] / w ** 3])


def _inv(M):
    """Inverse of small matrices: closed forms up to 3 x 3, LU beyond."""
    D = M.shape[-1]
    if D == 1:
        return 1 / M
    if D > 3:
        return torch.linalg.inv(M)
    if D == 2:
        adj = torch.stack([M[..., 1, 1], -M[..., 0, 1], -M[..., 1, 0], M[..., 0, 0]], -1).reshape(M.shape)
        return adj / (M[..., 0, 0] * M[..., 1, 1] - M[..., 0, 1] * M[..., 1, 0])[..., None, None]
    r = [M[..., i, :] for i in range(3)]
    cof = [torch.linalg.cross(r[1], r[2]), torch.linalg.cross(r[2], r[0]), torch.linalg.cross(r[0], r[1])]
    return torch.stack(cof, -1) / (r[0] * cof[0]).sum(-1)[..., None, None]


class _Block:
    """G on the correlated block by eliminating the other orbitals of every k, for chunks of frequencies."""

    def __init__(self, H, D):
        self.n, self.D, self.m = H.shape[1], D, H.shape[1] - D
        self.Hpp = H[:, :D, :D]
        if self.m:
            self.e, V = torch.linalg.eigh(H[:, D:, D:])
            b = H[:, :D, D:] @ V
            self.P = torch.einsum("kal,kbl->klab", b, b.conj()).reshape(H.shape[0], self.m, D * D)

    def chunk(self, f):
        return max(1, min(f, int(6e7 / (self.Hpp.shape[0] * max(self.D ** 2, self.m)))))

    def S(self, z, sig):
        """z - H_PP - sig - sum_l P_l/(z - e_l) [k, f, D, D] and 1/(z - e_l)."""
        D = self.D
        M = -self.Hpp[:, None] - sig[None] + z[None, :, None, None] * torch.eye(D, device=z.device)
        w = None
        if self.m:
            w = 1 / (z[None, :, None] - self.e[:, None, :])
            M = M - (w @ self.P).reshape(M.shape)
        return M, w


def _fermi(x, cut):
    f = torch.sigmoid(-x)
    return torch.where(x > 100, 0.0, torch.where(x < -100, 1.0, f)) if cut else f


def _exact_gloc(H, S, mu, beta, D):
    mom = _moments(S, beta)
    nf, nk = S.shape[0], H.shape[0]
    sig = _tail(S, beta, mom)
    m0 = torch.as_tensor(mom[0], device=H.device)
    w = _wn(2 * nf, beta, H.device)
    blk = _Block(H, D)
    step = blk.chunk(2 * nf)
    g, g0 = [], []
    for a in range(0, 2 * nf, step):
        M, _ = blk.S(mu + 1j * w[a:a + step], sig[a:a + step])
        g.append(_inv(M).mean(0))
        g0.append(_inv(M + sig[a:a + step] - m0).mean(0))
    g, g0 = torch.cat(g), torch.cat(g0)
    Hs = H.clone()
    Hs[:, :D, :D] += m0
    e0, U = torch.linalg.eigh(Hs)
    U = U[:, :D]
    occ = ((U * _fermi(beta * (e0 - mu), True)[:, None, :]) @ U.mH).mean(0)
    d = (g - g0).sum(0)
    return g[:nf], g0[:nf], (d + d.mH) / beta + occ


def _nele(blk, e0, sig, w, mu, beta):
    """N(mu) = (2/beta) sum_n Re[Tr G - Tr G0] + sum_l f(e0_l - mu), averaged over k."""
    tot, step = 0.0, blk.chunk(len(w))
    eye = torch.eye(blk.D, device=w.device)
    for a in range(0, len(w), step):
        z = mu + 1j * w[a:a + step]
        M, wl = blk.S(z, sig[a:a + step])
        X = _inv(M)
        if blk.m:
            tr = (X * (eye + ((wl * wl) @ blk.P).reshape(M.shape)).transpose(-1, -2)).sum((-1, -2)) + wl.sum(-1)
        else:
            tr = torch.einsum("...ii", X)
        tot += float((tr - (1 / (z[None, :, None] - e0[:, None])).sum(-1)).real.sum())
    return (2 / beta * tot + float(torch.sigmoid(-beta * (e0 - mu)).sum())) / blk.Hpp.shape[0]


def _exact_mu(c, H, S, mu):
    D, beta = c["D"], c["beta"]
    mom = _moments(S, beta)
    sig = _tail(S, beta, mom)
    nf2 = sig.shape[0]
    w = PI / beta + torch.arange(nf2, dtype=torch.float64, device=H.device) * (2 * PI / beta)
    Hs = H.clone()
    Hs[:, :D, :D] += torch.as_tensor(mom[0], device=H.device)
    e0 = torch.linalg.eigvalsh(Hs)
    blk, goal = _Block(H, D), _fill(c)
    N = lambda x: _nele(blk, e0, sig, w, x, beta)
    if c["newton"]:
        x, y = mu, N(mu)
        lo, hi = (x, None) if y < goal else (None, x)
        step = 0.1 if y < goal else -0.1
        for _ in range(60):
            nx = x + step
            if lo is not None and hi is not None and not lo < nx < hi:
                nx = (lo + hi) / 2
            ny = N(nx)
            lo, hi = (nx, hi) if ny < goal else (lo, nx)
            slope = (ny - y) / (nx - x)
            x, y = nx, ny
            if abs(ny - goal) < 1e-13 * goal:
                break
            step = (goal - ny) / slope if slope > 0 else math.copysign(0.5, goal - ny)
            if abs(step) < 1e-14:
                break
        return (x,)
    # the reference's bracket and bisection to |dmu| <= 1e-5
    evals, dmu = 1, 1.0
    cur, prev = N(mu), -1.0
    ub = lb = 0.0
    near = False
    if cur < goal:
        mu -= dmu + dmu
    while cur != goal and abs(dmu) > 1e-5:
        mu += dmu
        prev, cur = cur, N(mu)
        evals += 1
        if not near:
            if cur < goal:
                lb = mu
                if prev > goal and prev > 0:
                    near = True
                else:
                    dmu = abs(dmu)
            if cur > goal:
                ub = mu
                if prev < goal and prev > 0:
                    near = True
                else:
                    dmu = -abs(dmu)
        else:
            if cur > goal:
                ub = mu
            elif cur < goal:
                lb = mu
            dmu = (ub + lb) / 2 - mu
    return mu, evals


def _full(H, z, sig, D):
    """(z - H - sig on the correlated block)^-1 [k, f, n, n]."""
    M = -H[:, None].repeat(1, len(z), 1, 1)
    M[:, :, :D, :D] -= sig[None]
    M.diagonal(dim1=-2, dim2=-1).add_(z[None, :, None])
    return torch.linalg.inv(M)


def exact(case, seed):
    c, dev = case, torch.device("cuda", 0)
    kind = c["kind"]
    if kind in ("scgf2", "dmft"):
        return None
    if kind == "batch":
        return [list(exact({k: v for k, v in p.items() if k != "seed"}, p["seed"])) for p in _batch(c, seed)]
    if kind == "hk":
        rng = np.random.default_rng([int(seed), 1])
        R, T = _random_hoppings(rng, c["n"], c["rmax"], 0.5, np.linspace(-3, 0, c["n"]))
        return _hk(R, T, c["kx"], c["ky"], c["kz"], dev)
    R, T = _model(c, seed)
    H, S = _hk(R, T, c["kx"], c["ky"], c["kz"], dev), _sigma(c, seed, dev)
    rng = np.random.default_rng([int(seed), 4])
    mu, beta, D, nf = float(rng.uniform(-0.5, 0.5)), c["beta"], c["D"], c["nfreq"]
    if kind == "gloc":
        got = _exact_gloc(H, S, mu, beta, D)
        return [x.cpu().numpy() for x in got] if c.get("host") else list(got)
    if kind == "mu":
        return list(_exact_mu(c, H, S, mu))
    nk = H.shape[0]
    if kind == "derivs":
        sd = torch.as_tensor(rng.normal(size=(nf, D, D)) + 1j * rng.normal(size=(nf, D, D)), device=dev)
        md = float(rng.uniform(0.1, 1.0))
        z = mu + 1j * _wn(nf, beta, dev)
        step = max(1, int(2e8 / (nk * c["n"] ** 2 * 16)))
        gd, sb, mb = [], [], 0.0
        for a in range(0, nf, step):
            G = _full(H, z[a:a + step], S[a:a + step], D)
            g2 = G[..., :D, :] @ G[..., :, :D]
            G = G[..., :D, :D]
            x = (G @ sd[None, a:a + step] @ G - md * g2).mean(0)
            gd.append(x)
            sb.append((G.mH @ x[None] @ G.mH).mean(0))
            mb -= float((g2.mean(0).conj() * x).real.sum())
        return [torch.cat(gd), torch.cat(sb), mb]
    mom = _moments(S, beta)
    sig = _tail(S, beta, mom)
    z = mu + 1j * _wn(2 * nf, beta, dev)
    Hs = H.clone()
    Hs[:, :D, :D] += torch.as_tensor(mom[0], device=dev)
    e0, U = torch.linalg.eigh(Hs)
    step = max(1, int(4e8 / (nk * c["n"] ** 2 * 16)))
    tot = torch.zeros_like(H)
    for a in range(0, 2 * nf, step):
        G = _full(H, z[a:a + step], sig[a:a + step], D).sum(1)
        tot += G + G.mH
    r = sum(2 * (1 / (z[None, a:a + 256, None] - e0[:, None])).real.sum(1) for a in range(0, 2 * nf, 256))
    return tot / beta + (U * (_fermi(beta * (e0 - mu), True) - r / beta)[:, None, :]) @ U.mH
