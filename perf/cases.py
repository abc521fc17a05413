"""The work a user of the multi-sphere solver has it do, as cases that can be timed and checked.

Scenes are the repository's own kinds at generic sizes: the 64-sphere cluster (order 15), lognormal
water-sphere clusters at the number density of the 2000-sphere scene (per-sphere orders 9..30), hcp
clusters of 7.5 nm spheres (order 5, the smallest translations), long-wave clusters for the ML-FMM.
Coefficient vectors are compared in the basis x_nm / g_nm, g_nm = sqrt((n+m)!/(n-m)!), in which all
orders have comparable size (in the solver's own layout the entries of one sphere span 30 decades and
a norm would see the largest orders only).

exact() restates the coupling operator, the right-hand side and the field in plain torch, FP64: rotations
by the eigenvectors of J_y, Gaunt coefficients by Gauss-Legendre quadrature, GMRES without restarts.
"""
import math

import numpy as np
import torch

from itofoggysim_b200 import scene as S
from itofoggysim_b200 import server, solver

DEV = "cuda"


# ---- the cases -----------------------------------------------------------------------------------

def listed():
    return [
        # one operator application inside a user's own Krylov loop, device buffers.  Smallest
        # translations, where launches and latency count: an hcp half-sphere, coupling by j_n
        dict(name="operator-hcp-40", kind="operator", scene="hcp", size=40, z=1),
        # the 64-sphere cluster
        dict(name="operator-cluster-64", kind="operator", scene="cluster", size=64, z=3),
        # the flagship shape (lognormal radii, orders 11..28), the largest that fits three times
        dict(name="operator-lognormal-1000", kind="operator", scene="lognormal", size=1000, z=3),
        # scenes whose pair tables do not fit the memory sum the coaxial coefficients per application
        dict(name="operator-no-tables-211", kind="operator", scene="lognormal", size=211, z=3, pair_tables=-1),
        # several vectors at once from host arrays (a block method of the user's own)
        dict(name="operator-block-130x12", kind="operator_block", scene="lognormal", size=130, z=3, rhs=12),
        # the whole call: one plane wave, GMRES(30) to 1e-8, host to host
        dict(name="solve-cluster-64", kind="solve", scene="cluster", size=64, z=3, precision=0, tol=1e-8,
             restart=30),
        # mixed precision refined to a tight tolerance
        dict(name="solve-mixed-250", kind="solve", scene="lognormal", size=250, z=3, precision=1, tol=1e-11,
             restart=50),
        # many incidence directions and polarisations of one scene as a block, mixed precision
        dict(name="solve-block-mixed-64x32", kind="solve_block", scene="cluster", size=64, z=3, precision=1,
             tol=1e-11, restart=30, rhs=32),
        # a request of the serving stream: new geometry each time, so set-up and pair tables count
        dict(name="request-83x5", kind="request", scene="lognormal", size=83, z=3, precision=0, tol=1e-6,
             restart=30, rhs=5),
        # the ML-FMM operator with per-level orders
        dict(name="fmm-operator-2000", kind="operator", scene="longwave", size=2000, z=3, fmm_digits=3.0),
        # a whole solve through it
        dict(name="fmm-solve-500", kind="solve", scene="longwave", size=500, z=3, precision=0, tol=1e-8,
             restart=30, fmm_digits=3.0),
        # the field plot of an hcp cluster, 200 x 233 points from and to host arrays
        dict(name="field-hcp-71", kind="field", scene="hcp", size=71, z=1, nx=200, nz=233),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.choice(["operator", "operator", "operator", "no_tables", "operator_block", "solve", "solve_mixed",
                    "solve_block", "request", "fmm_operator", "fmm_solve", "field"])
    if k == "operator":
        sc = rng.choice(["hcp", "cluster", "lognormal", "lognormal"])
        size = {"hcp": _log(rng, 10, 125), "cluster": _log(rng, 8, 120), "lognormal": _log(rng, 8, 900)}[sc]
        c = dict(kind="operator", scene=sc, size=size, z=1 if sc == "hcp" else rng.choice([3, 3, 1]))
        if sc == "cluster":
            c["order"] = rng.randint(3, 20)
        return c
    if k == "no_tables":
        return dict(kind="operator", scene="lognormal", size=_log(rng, 20, 300), z=3, pair_tables=-1)
    if k == "operator_block":
        return dict(kind="operator_block", scene="lognormal", size=_log(rng, 20, 150), z=3, rhs=rng.randint(2, 20))
    if k == "solve":
        return dict(kind="solve", scene=rng.choice(["cluster", "lognormal"]), size=_log(rng, 12, 150), z=3,
                    precision=0, tol=rng.choice([1e-6, 1e-8, 1e-10]), restart=rng.choice([20, 30, 50]))
    if k == "solve_mixed":
        return dict(kind="solve", scene="lognormal", size=_log(rng, 20, 200), z=3, precision=1, tol=1e-11,
                    restart=rng.choice([30, 50]))
    if k == "solve_block":
        return dict(kind="solve_block", scene=rng.choice(["cluster", "lognormal"]), size=_log(rng, 16, 64), z=3,
                    precision=rng.choice([0, 1]), tol=1e-11, restart=30, rhs=rng.randint(2, 24))
    if k == "request":
        return dict(kind="request", scene="lognormal", size=_log(rng, 50, 100), z=3, precision=0, tol=1e-6,
                    restart=30, rhs=rng.randint(1, 8))
    if k == "fmm_operator":
        return dict(kind="operator", scene="longwave", size=_log(rng, 200, 2000), z=3,
                    fmm_digits=rng.choice([2.0, 3.0, 4.0]))
    if k == "fmm_solve":
        return dict(kind="solve", scene="longwave", size=_log(rng, 100, 500), z=3, precision=0, tol=1e-8, restart=30,
                    fmm_digits=3.0)
    return dict(kind="field", scene="hcp", size=_log(rng, 10, 125), z=1, nx=rng.randint(40, 200),
                nz=rng.randint(40, 233))


# ---- scenes ----------------------------------------------------------------------------------------

def _waves(nr, rng):
    """nr plane waves: one along +z, or random directions with alternating polarisation."""
    if nr == 1:
        return S.single_wave()
    th = np.arccos(rng.uniform(-1.0, 1.0, nr))
    jones = np.tile([[1.0, 0.0, 0.0, 0.0], [0.0, 0.0, 1.0, 0.0]], ((nr + 1) // 2, 1))[:nr]
    return dict(wave_theta=th, wave_phi=rng.uniform(0.0, 2.0 * math.pi, nr), jones=jones, wave_g=np.ones(nr),
                wave_phase=np.zeros(nr), wave_d0=np.zeros((nr, 3)))


def _scene(case, seed):
    rng = np.random.default_rng(seed)
    n = case["size"]
    kw = dict(z_coupling=case["z"], gmres_restart=case.get("restart", 30), gmres_tolerance=case.get("tol", 1e-8),
              reference_row_rule=False, waves=_waves(case.get("rhs", 1), rng))
    if case["scene"] == "cluster":
        # r = 0.5 um at the number density of 64 in a 10 um cube
        return S.make_scene(np.full(n, 0.5), 10.0 * (n / 64.0) ** (1.0 / 3.0), seed, n_max=case.get("order"), **kw)
    if case["scene"] == "lognormal":
        # the size distribution belongs to the case (it sets the orders, so the vectors' lengths)
        radii = S.lognormal_radii(np.random.default_rng(1000 + n), n)
        return S.make_scene(radii, 40.0 * (n / 2000.0) ** (1.0 / 3.0), seed, **kw)
    if case["scene"] == "longwave":
        return S.make_scene(rng.uniform(0.1, 0.3, n), (n / 0.04) ** (1.0 / 3.0), seed, lambda_0=6.0, n_max=8, **kw)
    # the first `size` sites of an hcp half-sphere, each moved by up to 0.1 nm
    radius = 0.02
    while True:
        sc = S.hcp_sphere_scene(radius)
        if sc.n_spheres >= n:
            break
        radius += 0.001
    c = sc.centres[:n] + rng.uniform(-1e-4, 1e-4, (n, 3)) / math.sqrt(3.0)
    sc.centres = np.ascontiguousarray(c)
    sc.param_index = np.zeros(n, np.int32)
    return sc


def _g(sc):
    """g_nm over the solver's vector layout (|g|; its sign (-1)^m is kept out of the scaling)."""
    g = np.array([math.sqrt(math.factorial(n + m) / math.factorial(n - m))
                  for n in range(1, sc.n_range[1] + 1) for m in range(-n, n + 1)])
    return np.tile(g, 2 * sc.n_spheres)


def _vector(sc, seed, nr=None):
    """Random coefficients of unit size in the scaled basis, zero above each sphere's own order."""
    p = torch.as_tensor(sc.p_of_sphere().astype(np.int64), device=DEV)
    deg = torch.as_tensor([n for n in range(1, sc.n_range[1] + 1) for _ in range(2 * n + 1)], device=DEV)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    shape = (nr or 1, sc.n_spheres, 2, deg.numel())
    x = torch.complex(torch.randn(shape, dtype=torch.float64, device=DEV, generator=gen),
                      torch.randn(shape, dtype=torch.float64, device=DEV, generator=gen))
    x = x * (deg[None, :] <= p[:, None])[None, :, None, :]
    return x.reshape(nr, -1) if nr else x.reshape(-1)


def _grid(sc, case):
    ext = 1.5 * float(np.abs(sc.centres).max() + sc.radius.max())
    X, Z = np.meshgrid(np.linspace(-ext, ext, case["nx"]), np.linspace(-ext, 1.3 * ext, case["nz"]), indexing="ij")
    return np.stack([X, np.zeros_like(X), Z], axis=-1).reshape(-1, 3)


# ---- prepare and run ---------------------------------------------------------------------------------

def prepare(case, seed):
    sc = _scene(case, seed)
    st = dict(case=case, sc=sc)
    kind = case["kind"]
    g = _g(sc)
    st["ginv"] = 1.0 / g
    if kind == "request":
        st["server"] = server.SolveServer(max_concurrent=2)
        return st
    kw = dict(precision=case.get("precision", 0), pair_tables=case.get("pair_tables", 0))
    if "fmm_digits" in case:
        kw.update(use_ml_fmm=True, fmm_convention=1, fmm_digits=case["fmm_digits"])
    st["solver"] = solver.MultiSphereSolver(sc, **kw)
    if kind == "operator":
        st["ginv"] = torch.as_tensor(1.0 / g, device=DEV)
        st["x"] = _vector(sc, seed) * torch.as_tensor(g, device=DEV)
        st["y"] = torch.empty_like(st["x"])
    elif kind == "operator_block":
        st["x"] = _vector(sc, seed, case["rhs"]).cpu().numpy() * g
    elif kind == "field":
        st["x"] = _vector(sc, seed).cpu().numpy() * 1e-6
        st["points"] = _grid(sc, case)
    torch.cuda.synchronize()
    return st


def run(st):
    kind = st["case"]["kind"]
    if kind == "operator":
        # the solver works on its own stream: what this stream still does with the buffers ends first
        torch.cuda.current_stream().synchronize()
        st["solver"].matvec_device(st["x"].data_ptr(), st["y"].data_ptr())
        return st["y"] * st["ginv"]
    if kind == "operator_block":
        return st["solver"].calculate_vector_b_block(st["x"]) * st["ginv"]
    if kind == "solve":
        x, _ = st["solver"].solve()
        return x * st["ginv"]
    if kind == "solve_block":
        x, cs, _, _, _ = st["solver"].solve_block()
        return {"x": x * st["ginv"], "cross_sections": cs}
    if kind == "request":
        srv = st["server"]
        rid = srv.submit(st["sc"], rhs_per_wave=True, precision=st["case"]["precision"])
        info, x, cs = srv.wait(rid)
        srv.release(rid)
        if x is None:
            raise RuntimeError(info["error"])
        return {"x": x * st["ginv"], "cross_sections": cs}
    E, H = st["solver"].get_field(st["x"], st["points"])
    return {"E": E, "H": H}


# ---- work --------------------------------------------------------------------------------------------

def _pair_flops(sc):
    """Flops of one operator application: per ordered pair two rotations (real d-matrix times complex
    vector, both ways, two parts) and the axial step (four complex multiply-adds per entry)."""
    cnt = np.bincount(sc.p_of_sphere())
    tot = 0.0
    for a in np.nonzero(cnt)[0]:
        for b in np.nonzero(cnt)[0]:
            rot = sum((2 * n + 1) ** 2 for n in range(1, a + 1)) + sum((2 * n + 1) ** 2 for n in range(1, b + 1))
            ax = sum((a - max(1, abs(k)) + 1) * (b - max(1, abs(k)) + 1) for k in range(-min(a, b), min(a, b) + 1))
            tot += (cnt[a] * cnt[b] - (cnt[a] if a == b else 0)) * (8.0 * rot + 32.0 * ax)
    return tot


def work(case):
    sc = _scene(case, 1)
    vec = 16.0 * sc.vector_length()
    if case["kind"] == "field":
        pts = case["nx"] * case["nz"]
        P = sc.n_range[1] * (sc.n_range[1] + 2)
        return {"bytes": vec + pts * (24 + 96), "flops": pts * sc.n_spheres * P * 60.0}
    if case["scene"] == "longwave":
        # the ML-FMM's near field: about 27 leaf boxes of 10 spheres, and as much again for its boxes
        flops = _pair_flops(sc) / sc.n_spheres * min(sc.n_spheres, 540)
    else:
        flops = _pair_flops(sc)
    rhs = case.get("rhs", 1)
    its = 1
    if case["kind"] in ("solve", "solve_block", "request"):
        # Arnoldi steps that a solve to the tolerance needs at these densities
        its = int(3 + 2.5 * -math.log10(case["tol"]))
    return {"bytes": 2 * vec * rhs * its, "flops": float(flops * rhs * its)}


# ---- the same in plain torch, 64 bits ------------------------------------------------------------------

_C = torch.complex128


def _zbessel(z, rho, P):
    """[len(rho), P + 1] spherical Bessel function z_n(rho): 1 j_n, 3 h_n^(1)."""
    r = rho.cpu().numpy()
    out = np.zeros((len(r), P + 1), complex)
    start = int(P + 40 + 1.2 * r.max())
    f1, f0 = np.zeros(len(r)), np.full(len(r), 1e-300)
    j = np.zeros((len(r), P + 2))
    for n in range(start, 0, -1):
        f1, f0 = f0, (2 * n + 1) / r * f0 - f1
        if n - 1 <= P + 1:
            j[:, n - 1] = f0
        big = np.abs(f0) > 1e200
        if big.any():
            f0[big] *= 1e-200
            f1[big] *= 1e-200
            j[big] *= 1e-200
    j0, j1 = np.sin(r) / r, (np.sin(r) / r - np.cos(r)) / r
    first = np.abs(j0) >= np.abs(j1)
    j *= np.where(first, j0 / np.where(first, j[:, 0], 1.0), j1 / np.where(first, 1.0, j[:, 1]))[:, None]
    # upward where that is the stable direction
    up = r > P + 1
    if up.any():
        ru = r[up]
        a, b = j0[up], j1[up]
        j[up, 0] = a
        for n in range(1, P + 2):
            j[up, n] = b
            a, b = b, (2 * n + 1) / ru * b - a
    out[:] = j[:, :P + 1]
    if z == 3:
        a, b = -np.cos(r) / r, (-np.cos(r) / r - np.sin(r)) / r
        for n in range(P + 1):
            out[:, n] += 1j * a
            a, b = b, (2 * n + 3) / r * b - a
    return torch.as_tensor(out, device=DEV)


def _legendre_hat(P, x):
    """{k: [P + 1, len(x)]} sqrt((n-k)!/(n+k)!) P_n^k(x) without the Condon-Shortley phase."""
    s = np.sqrt(1.0 - x * x)
    out = {}
    for k in range(P + 1):
        v = np.zeros((P + 1, len(x)))
        q = np.ones(len(x))
        for i in range(1, k + 1):
            q = q * math.sqrt((2.0 * i - 1.0) / (2.0 * i)) * s
        v[k] = q
        for n in range(k + 1, P + 1):
            v[n] = ((2 * n - 1) * x * v[n - 1]
                    - (math.sqrt((n - 1.0 - k) * (n - 1.0 + k)) * v[n - 2] if n >= k + 2 else 0.0)) \
                / math.sqrt((n - k) * (n + k))
        out[k] = v
    return out


class _Coupling:
    """sum_l [A x_a + B x_b ; B x_a + A x_b](k (d_l - d_j)) of a scene, scaled basis."""

    def __init__(self, sc):
        self.sc = sc
        self.p = sc.p_of_sphere().astype(int)
        self.pg = int(sc.n_range[1])
        M = int(self.p.max())
        # eigenvectors of J_y per degree: d(theta) = V exp(-i theta m) V^H
        self.V, self.m = {}, {}
        for n in range(1, M + 1):
            m = np.arange(-n, n + 1)
            up = np.diag(np.sqrt(n * (n + 1.0) - m[:-1] * (m[:-1] + 1.0)), -1)
            w, V = np.linalg.eigh((up - up.T) / 2j)
            self.V[n] = torch.as_tensor(V, device=DEV)
            self.m[n] = torch.as_tensor(np.round(w), device=DEV)
        # Gaunt coefficients (n mu p; -k k 0)(n mu p; 0 0 0)(2p+1) i^p for n, mu <= M + 1, by quadrature
        xq, wq = np.polynomial.legendre.leggauss(2 * M + 6)
        Ph = _legendre_hat(M + 1, xq)
        Pp = np.zeros((2 * M + 3, len(xq)))
        Pp[0], Pp[1] = 1.0, xq
        for q in range(2, 2 * M + 3):
            Pp[q] = ((2 * q - 1) * xq * Pp[q - 1] - (q - 1) * Pp[q - 2]) / q
        a = np.arange(M + 2)
        q = np.arange(2 * M + 3)
        tri = (q >= abs(a[:, None, None] - a[None, :, None])) & (q <= a[:, None, None] + a[None, :, None]) \
            & ((a[:, None, None] + a[None, :, None] + q) % 2 == 0)
        self.G = []
        for k in range(M + 1):
            G = np.einsum("aq,bq,pq->abp", Ph[k] * (0.5 * wq), Ph[k], Pp, optimize=True) * (2 * q + 1) * (-1) ** k
            self.G.append(torch.as_tensor((G * tri * (1j ** (q % 4)))[k:, k:], device=DEV))
        self.cen = torch.as_tensor(sc.centres, device=DEV)
        self.kept = None

    def _groups(self, chunk):
        """(target order, source order, targets, sources) of all ordered pairs, in chunks."""
        for a in np.unique(self.p):
            ta = np.nonzero(self.p == a)[0]
            for b in np.unique(self.p):
                sb = np.nonzero(self.p == b)[0]
                T, L = np.meshgrid(ta, sb, indexing="ij")
                T, L = T.reshape(-1), L.reshape(-1)
                ok = T != L
                T, L = T[ok], L[ok]
                for i in range(0, len(T), chunk):
                    yield int(a), int(b), torch.as_tensor(T[i:i + chunk], device=DEV), \
                        torch.as_tensor(L[i:i + chunk], device=DEV)

    def _geometry(self, a, b, T, L):
        d = self.sc.wavenumber * (self.cen[L] - self.cen[T])
        rho = d.norm(dim=1)
        th = torch.acos(d[:, 2] / rho)
        ph = torch.atan2(d[:, 1], d[:, 0])
        zeta = _zbessel(int(self.sc.z_coupling), rho, a + b + 1)
        # S(k; n, mu), n = k..a, mu = k..b + 1
        Sk = [torch.einsum("abp,up->uab", self.G[k][:a + 1 - k, :b + 2 - k, :a + b + 2], zeta)
              for k in range(min(a, b) + 1)]
        return rho, th, ph, Sk

    def _apply(self, a, b, T, L, geo, x, y):
        rho, th, ph, Sk = geo
        nr = x.shape[0]
        u = len(T)
        src = x[:, L]                                    # [nr, u, 2, C]
        km = min(a, b)
        xs = torch.zeros(nr, u, 2, b + 1, 2 * km + 1, dtype=_C, device=DEV)     # degree, order -km..km
        for n in range(1, b + 1):
            o = n * n - 1
            mu = torch.arange(-n, n + 1, device=DEV)
            v = src[..., o:o + 2 * n + 1] * torch.exp(1j * ph[:, None] * mu)[None, :, None, :]
            V, m = self.V[n], self.m[n]
            # x'(k) = sum_mu d_{mu k} x_mu = conj(V) exp(-i theta m) V^T
            v = (v @ V) * torch.exp(-1j * th[:, None] * m)[None, :, None, :]
            v = v @ V.conj().T
            w = min(n, km)
            xs[..., n, km - w:km + w + 1] = v[..., n - w:n + w + 1]
        ys = torch.zeros(nr, u, 2, a + 1, 2 * km + 1, dtype=_C, device=DEV)
        for k in range(km + 1):
            lo = max(1, k)
            n = torch.arange(lo, a + 1, device=DEV, dtype=torch.float64)
            nu = torch.arange(lo, b + 1, device=DEV, dtype=torch.float64)
            pre = (-1.0) ** k * (2 * nu + 1)[None, :] / (2 * n * (n + 1))[:, None]
            r = lo - k
            S0 = Sk[k][:, r:, r:b + 1 - k]
            Sp = Sk[k][:, r:, r + 1:b + 2 - k]
            if r > 0:
                Sm = Sk[k][:, r:, r - 1:b - k]
            else:
                Sm = torch.cat([torch.zeros_like(S0[:, :, :1]), S0[:, :, :-1]], dim=2)   # S(k; n, k - 1) = 0
            c1 = rho[:, None] * (2 * nu * torch.sqrt((nu + 1) ** 2 - k * k) / (2 * nu + 1))
            c2 = rho[:, None] * (2 * (nu + 1) * torch.sqrt(nu * nu - k * k) / (2 * nu + 1))
            A = pre * (2 * nu * (nu + 1) * S0 + 1j * (c1[:, None, :] * Sp - c2[:, None, :] * Sm))
            B = pre * 2j * k * rho[:, None, None] * S0
            for sg in ((1, -1) if k else (1,)):
                xa, xb = xs[:, :, 0, lo:, km + sg * k], xs[:, :, 1, lo:, km + sg * k]
                ys[:, :, 0, lo:, km + sg * k] = torch.einsum("uns,rus->run", A, xa) + sg * torch.einsum("uns,rus->run", B, xb)
                ys[:, :, 1, lo:, km + sg * k] = sg * torch.einsum("uns,rus->run", B, xa) + torch.einsum("uns,rus->run", A, xb)
        out = torch.zeros(nr, u, 2, self.pg * (self.pg + 2), dtype=_C, device=DEV)
        for n in range(1, a + 1):
            o = n * n - 1
            w = min(n, km)
            v = torch.zeros(nr, u, 2, 2 * n + 1, dtype=_C, device=DEV)
            v[..., n - w:n + w + 1] = ys[..., n, km - w:km + w + 1]
            V, m = self.V[n], self.m[n]
            v = (v @ V.conj()) * torch.exp(-1j * th[:, None] * m)[None, :, None, :]
            v = v @ V.T
            mm = torch.arange(-n, n + 1, device=DEV)
            out[..., o:o + 2 * n + 1] = v * torch.exp(-1j * ph[:, None] * mm)[None, :, None, :]
        y.index_add_(1, T, out)

    def apply(self, x, keep=False):
        """x [nr, spheres, 2, C] -> the same of the sums."""
        y = torch.zeros_like(x)
        if keep and self.kept is None:
            self.kept = [(a, b, T, L, self._geometry(a, b, T, L)) for a, b, T, L in self._groups(8192)]
        if self.kept is not None:
            chunk = max(16, 8192 // x.shape[0])
            for a, b, T, L, (rho, th, ph, Sk) in self.kept:
                for i in range(0, len(T), chunk):
                    q = slice(i, i + chunk)
                    self._apply(a, b, T[q], L[q], (rho[q], th[q], ph[q], [s[q] for s in Sk]), x, y)
        else:
            for a, b, T, L in self._groups(max(16, 8192 // x.shape[0])):
                self._apply(a, b, T, L, self._geometry(a, b, T, L), x, y)
        return y


def _mie(sc):
    """a_n, b_n of every sphere as [spheres, 2, C] factors."""
    pg = int(sc.n_range[1])
    tab = np.zeros((sc.n_param, 2, pg + 1), complex)
    for i in range(sc.n_param):
        x = sc.wavenumber * float(sc.radius[i])
        m = complex(sc.refractive_index[i]) / sc.n_medium
        p = min(int(sc.n_range_param[i, 1]), pg)
        z = m * x
        D = np.zeros(p + 60 + int(abs(z)) * 2, complex)
        for n in range(len(D) - 1, 0, -1):
            D[n - 1] = n / z - 1.0 / (D[n] + n / z)
        h = _zbessel(3, torch.tensor([x], dtype=torch.float64), p)[0].cpu().numpy()
        j = h.real
        for n in range(1, p + 1):
            for c, f in ((0, D[n] / m + n / x), (1, m * D[n] + n / x)):
                tab[i, c, n] = (f * j[n] - j[n - 1]) / (f * h[n] - h[n - 1])
    deg = np.array([n for n in range(1, pg + 1) for _ in range(2 * n + 1)])
    return torch.as_tensor(tab[sc.param_index][:, :, deg], device=DEV)


def _incident(sc):
    """[waves, spheres, 2, C] plane-wave coefficients p, q in the scaled basis (with g's sign (-1)^m)."""
    pg = int(sc.n_range[1])
    out = np.zeros((sc.n_waves, sc.n_spheres, 2, pg * (pg + 2)), complex)
    for w in range(sc.n_waves):
        al, be = float(sc.wave_theta[w]), float(sc.wave_phi[w])
        ca, sa = math.cos(al), math.sin(al)
        kv = sc.wavenumber * np.array([sa * math.cos(be), sa * math.sin(be), ca])
        e = np.exp(1j * ((sc.centres - sc.wave_d0[w]) @ kv + sc.wave_phase[w]))
        pi, tau = np.zeros(pg * (pg + 2)), np.zeros(pg * (pg + 2))
        for m in range(pg + 1):
            mq = max(m, 1)
            q = np.zeros(pg + 1)          # sqrt((n-mq)!/(n+mq)!) P_n^mq / sin
            v = 1.0
            for i in range(1, mq + 1):
                v *= math.sqrt((2.0 * i - 1.0) / (2.0 * i))
            q[mq:mq + 1] = v * sa ** (mq - 1)
            for n in range(mq + 1, pg + 1):
                q[n] = ((2 * n - 1) * ca * q[n - 1]
                        - (math.sqrt((n - 1.0 - mq) * (n - 1.0 + mq)) * q[n - 2] if n >= mq + 2 else 0.0)) \
                    / math.sqrt((n - mq) * (n + mq))
            for n in range(mq, pg + 1):
                o = n * n - 1 + n
                if m == 0:
                    tau[o] = -math.sqrt(n * (n + 1.0)) * sa * q[n]
                    continue
                t = n * ca * q[n] - math.sqrt((n + m) * (n - m)) * q[n - 1]
                s = (-1.0) ** m
                pi[o + m], tau[o + m] = s * m * q[n], s * t
                pi[o - m], tau[o - m] = -m * q[n], t
        deg = np.array([n for n in range(1, pg + 1) for _ in range(2 * n + 1)])
        mm = np.array([m for n in range(1, pg + 1) for m in range(-n, n + 1)])
        base = np.exp(-1j * mm * be) / (deg * (deg + 1.0))
        jx = complex(sc.jones[w, 0], sc.jones[w, 1])
        jy = complex(sc.jones[w, 2], sc.jones[w, 3])
        f = sc.wave_g[w] * e[:, None]
        out[w, :, 0] = f * base * (jx * tau + jy * pi)
        out[w, :, 1] = f * base * (jx * pi + jy * tau)
    return torch.as_tensor(out, device=DEV)


def _sign(sc):
    """(-1)^m over [C]: the solver's g_nm carries it, the scaling of the outputs does not."""
    return torch.as_tensor([(-1.0) ** m for n in range(1, sc.n_range[1] + 1) for m in range(-n, n + 1)],
                           dtype=torch.float64, device=DEV)


def _gmres(op, b):
    """Full GMRES for a batch of right-hand sides [nr, n] down to rounding."""
    beta = b.norm(dim=1)
    V = [b / beta[:, None]]
    nr = b.shape[0]
    steps = 200
    H = torch.zeros(nr, steps + 1, steps, dtype=_C, device=DEV)
    x = None
    for k in range(steps):
        w = op(V[k])
        for _ in range(2):
            for i in range(k + 1):
                h = (V[i].conj() * w).sum(dim=1)
                H[:, i, k] += h
                w = w - h[:, None] * V[i]
        nw = w.norm(dim=1)
        H[:, k + 1, k] = nw
        V.append(w / nw[:, None])
        if k % 5 == 4 or k == steps - 1:
            rhs = torch.zeros(nr, k + 2, 1, dtype=_C, device=DEV)
            rhs[:, 0, 0] = beta
            Hk = H[:, :k + 2, :k + 1]
            Q, R = torch.linalg.qr(Hk, mode="reduced")
            yk = torch.linalg.solve_triangular(R, Q.mH @ rhs, upper=True)
            res = (rhs - Hk @ yk).norm(dim=(1, 2)) / beta
            if float(res.max()) < 3e-15 or k == steps - 1:
                x = sum(yk[:, i] * V[i] for i in range(k + 1))
                break
    return x


def exact(case, seed):
    sc = _scene(case, seed)
    kind = case["kind"]
    pg, N = int(sc.n_range[1]), sc.n_spheres
    C = pg * (pg + 2)
    sgn = _sign(sc)
    if kind == "field":
        return _field(sc, case, _vector(sc, seed).cpu().numpy() * 1e-6)
    if kind in ("solve", "solve_block") and sc.ragged_unknowns() * case.get("rhs", 1) > 2_500_000:
        return None      # the kept geometry and the Krylov bases would take over 20 seconds
    cp = _Coupling(sc)
    mie = _mie(sc)
    if kind in ("operator", "operator_block"):
        x = _vector(sc, seed, case.get("rhs")).reshape(-1, N, 2, C)
        y = x + mie * cp.apply(x * sgn) * sgn
        return y.reshape(-1) if kind == "operator" else y.reshape(-1, N * 2 * C).cpu().numpy()
    # a solve: one right-hand side per wave, or the waves' sum
    inc = _incident(sc)
    if kind == "solve":
        inc = inc.sum(dim=0, keepdim=True)
    nr = inc.shape[0]
    b = mie * inc

    def op(v):
        v = v.reshape(nr, N, 2, C)
        return (v + mie * cp.apply(v, keep=True)).reshape(nr, -1)

    x = _gmres(op, b.reshape(nr, -1)).reshape(nr, N, 2, C)
    out = (x * sgn).reshape(nr, -1).cpu().numpy()
    if kind == "solve":
        return out[0]
    n = torch.as_tensor([v for v in range(1, pg + 1) for _ in range(2 * v + 1)], dtype=torch.float64, device=DEV)
    wt = n * (n + 1) * (2 * n + 1)
    ext = (wt * (inc.conj() * x).real).sum(dim=(1, 2, 3))
    inv = torch.where(mie != 0, (1.0 / torch.where(mie != 0, mie, torch.ones_like(mie))).real - 1.0,
                      torch.zeros_like(mie.real))
    ab = (wt * x.abs() ** 2 * inv).sum(dim=(1, 2, 3))
    f = 4.0 * math.pi / sc.wavenumber ** 2
    cs = torch.stack([f * (ext - ab), f * ext, f * ab], dim=1).cpu().numpy()
    return {"x": out, "cross_sections": cs}


def _field(sc, case, x):
    """E, H of the outgoing expansions at the grid points, zero inside a sphere."""
    pts = torch.as_tensor(_grid(sc, case), device=DEV)
    pg = int(sc.n_range[1])
    C = pg * (pg + 2)
    x = torch.as_tensor(x.reshape(sc.n_spheres, 2, C), device=DEV)
    E = torch.zeros(len(pts), 3, dtype=_C, device=DEV)
    H = torch.zeros_like(E)
    inside = torch.zeros(len(pts), dtype=torch.bool, device=DEV)
    for j in range(sc.n_spheres):
        d = pts - torch.as_tensor(sc.centres[j], device=DEV)
        r = d.norm(dim=1)
        inside |= ~(r > float(sc.radius[sc.param_index[j]]))
        r = torch.where(r > 0, r, torch.ones_like(r))
        ct = d[:, 2] / r
        th = torch.acos(ct)
        ct, st = torch.cos(th), torch.sin(th)
        ph = torch.atan2(d[:, 1], d[:, 0])
        rho = sc.wavenumber * r
        h = _zbessel(3, rho, pg + 1)
        es = torch.zeros(len(pts), 3, dtype=_C, device=DEV)
        hs = torch.zeros_like(es)
        for m in range(pg + 1):
            mq = max(m, 1)
            q = [torch.zeros_like(ct) for _ in range(pg + 1)]
            P = [torch.zeros_like(ct) for _ in range(pg + 1)]
            v = 1.0
            for i in range(1, mq + 1):
                v *= 2.0 * i - 1.0
            if mq <= pg:
                q[mq] = v * st ** (mq - 1)
            P[m] = q[m] * st if m else torch.ones_like(ct)
            for n in range(mq + 1, pg + 1):
                q[n] = ((2 * n - 1) * ct * q[n - 1] - (n + mq - 1) * q[n - 2]) / (n - mq)
            for n in range(m + 1, pg + 1):
                P[n] = ((2 * n - 1) * ct * P[n - 1] - (n + m - 1) * (P[n - 2] if n >= 2 else 0.0)) / (n - m)
            for n in range(mq, pg + 1):
                xi = 0.5 * (rho * h[:, n - 1] + h[:, n] - rho * h[:, n + 1])
                ratio = math.factorial(n - m) / math.factorial(n + m)
                for s in ((1, -1) if m else (1,)):
                    f = 1.0 if s == 1 else (-1.0) ** m * ratio
                    pi = s * m * q[n] * f
                    tau = -st * q[n] if m == 0 else f * (n * ct * q[n] - (n + m) * q[n - 1])
                    e = torch.exp(1j * s * m * ph)
                    Mt, Mp = 1j * pi * h[:, n] * e, -tau * h[:, n] * e
                    Nr = n * (n + 1) * (f * P[n]) / rho * h[:, n] * e
                    Nt, Np = tau / rho * xi * e, 1j * pi / rho * xi * e
                    Enm = (1j ** n) * (2 * n + 1) * (ratio if s == 1 else 1.0 / ratio)
                    an, bn = x[j, 0, n * n - 1 + n + s * m], x[j, 1, n * n - 1 + n + s * m]
                    es += (1j * Enm) * torch.stack([an * Nr, an * Nt + bn * Mt, an * Np + bn * Mp], dim=1)
                    hs += Enm * torch.stack([bn * Nr, bn * Nt + an * Mt, bn * Np + an * Mp], dim=1)
        cp, sp = torch.cos(ph), torch.sin(ph)
        for out, v, f in ((E, es, 1.0), (H, hs, sc.n_medium / 299792458.0)):
            out[:, 0] += f * (st * cp * v[:, 0] + ct * cp * v[:, 1] - sp * v[:, 2])
            out[:, 1] += f * (st * sp * v[:, 0] + ct * sp * v[:, 1] + cp * v[:, 2])
            out[:, 2] += f * (ct * v[:, 0] - st * v[:, 1])
    E[inside] = 0
    H[inside] = 0
    return {"E": E.cpu().numpy(), "H": H.cpu().numpy()}
