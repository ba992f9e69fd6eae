"""The work this framework's users have it do, as measurable cases.

A case is a dict of plain values; `prepare` builds what a program holds before
the call (inputs on the GPU or, for the drop-ins, on the host, and the engine it
keeps), `run` is one pass through the public entry points, `exact` the same
result from plain torch FFTs in FP64, `work` the bytes and operations a pass
cannot do without.

Kinds:
  ns3d      a 3D engine (Navier-Stokes RK4/CN or Heun/CN, Euler, Boussinesq): a
            state on the device is uploaded, stepped and downloaded
  bous_abi  the Boussinesq `timestep_cuda_` on page-locked host arrays, advanced in
            place as the reference's drivers do
  ns2d_abi  the 2D `timestep_cuda_` on a host array
  batch2d   independent 2D runs of mixed sizes in one launch, advanced in place
  tangent2d an exact Jacobian-vector product over a period (Floquet, Krylov)
  newton2d  one Newton-GMRES-hookstep iteration of a batch of UPO guesses
  adjoint3d a gradient through a 3D trajectory (forward and backward)
"""
import math

import numpy as np
import torch

import psgpu_b200 as P
from psgpu_b200 import abi, adjoint
from psgpu_b200.fields import Grid2D, Grid3D

SCHEMES = {"heun": P.SCHEME_NS_HEUN, "euler": P.SCHEME_EULER_HEUN, "rk4": P.SCHEME_NS_RK4,
           "bous": P.SCHEME_BOUS_RK4}


def _ns3d(name, scheme, n, prec, steps, nu=1 / 400, dt=2e-3, ampfor=0.0, kf=4, ri=0.0, theta=0.0):
    c = {"kind": "ns3d", "scheme": scheme, "n": n, "prec": prec, "steps": steps, "nu": nu, "dt": dt,
         "ampfor": ampfor, "kf": kf, "ri": ri, "theta": theta}
    return dict(name=name, **c) if name else c


def listed():
    return [
        # the headline run: FP32 256^3 RK4/CN between two outputs of a DNS
        _ns3d("ns3d_rk4_f32_256", "rk4", 256, 32, 10, nu=1 / 1600, dt=1e-3),
        # the smallest 3D call: one step of a toy grid, all launch latency
        _ns3d("ns3d_rk4_f32_32", "rk4", 32, 32, 1, dt=5e-3),
        # the reference's precision at the grid its build is set to
        _ns3d("ns3d_rk4_f64_128", "rk4", 128, 64, 3),
        # the forced DNS build's scheme at that grid
        _ns3d("ns3d_heun_f64_128", "heun", 128, 64, 5, ampfor=0.05),
        # stratified flow at the headline grid, gravity along z
        _ns3d("bous_f32_256", "bous", 256, 32, 3, nu=1 / 1600, dt=1e-3, ri=1.0),
        # the Boussinesq driver's call: host arrays in, nine steps and the half step that
        # ends its interval, host arrays out
        {"name": "bous_abi_f64_128", "kind": "bous_abi", "n": 128, "steps": 10, "nu": 1 / 400,
         "dt": 1e-3, "ri": 1.0, "theta": 0.3},
        # the 2D driver's call: one period-sized integration of one state
        {"name": "ns2d_abi_f64_128", "kind": "ns2d_abi", "n": 128, "steps": 200, "nu": 1 / 40,
         "dt": 0.005},
        # the ensemble: uneven sizes, FP32, a short span between recurrence checks
        {"name": "batch2d_f32_mixed", "kind": "batch2d", "sizes": "64,128,256", "count": 384,
         "prec": 32, "steps": 10, "dt": 0.005},
        # the smallest 2D call: one small run, a few steps
        {"name": "batch2d_f64_one_32", "kind": "batch2d", "sizes": "32", "count": 1, "prec": 64,
         "steps": 5, "dt": 0.005},
        # one Floquet / Krylov product over a short period
        {"name": "tangent2d_f64_128", "kind": "tangent2d", "n": 128, "period": 0.503, "nu": 1 / 40,
         "dt": 0.005},
        # a Newton iteration of a dozen guesses of uneven periods (the whole solver: some 40
        # Krylov products in lock step, then the hookstep's trials)
        {"name": "newton2d_64", "kind": "newton2d", "n": 64, "guesses": 12, "kmax": 60,
         "tmin": 1.0, "tmax": 2.0, "nu": 1 / 20, "dt": 0.0125, "gmtol": 0.1},
        # the gradient study's call: forward with checkpoints, backward
        {"name": "adjoint3d_f64_64", "kind": "adjoint3d", "n": 64, "prec": 64, "steps": 7,
         "every": 4, "nu": 1 / 200, "dt": 5e-3},
    ]


def draw(rng):
    kind = rng.choice(["ns3d", "ns3d", "ns3d", "batch2d", "batch2d", "ns2d_abi", "tangent2d", "adjoint3d"])
    prec = rng.choice([32, 64])
    nu = math.exp(rng.uniform(math.log(1 / 1600), math.log(1 / 50)))
    if kind == "ns3d":
        n = rng.choice([16, 32, 64, 128, 256])
        most = {16: 40, 32: 40, 64: 30, 128: 15, 256: 4}[n]
        steps = int(round(math.exp(rng.uniform(0, math.log(most)))))
        scheme = rng.choice(["rk4", "heun", "euler", "bous"])
        return _ns3d(None, scheme, n, prec, steps, nu=nu, dt=rng.uniform(5e-4, 2e-3),
                     ampfor=rng.choice([0.0, 0.05]) if scheme != "euler" else 0.0,
                     kf=rng.choice([1, 2, 4]), ri=rng.uniform(0.1, 2.0) if scheme == "bous" else 0.0,
                     theta=rng.uniform(0.0, 1.5) if scheme == "bous" else 0.0)
    if kind == "batch2d":
        sizes = rng.sample([16, 32, 64, 128, 256], rng.randint(1, 4))
        count = int(round(math.exp(rng.uniform(0, math.log(300)))))
        return {"kind": "batch2d", "sizes": ",".join(map(str, sorted(sizes))), "count": count,
                "prec": prec, "steps": rng.randint(1, 12), "dt": rng.uniform(2e-3, 6e-3)}
    if kind == "ns2d_abi":
        return {"kind": "ns2d_abi", "n": rng.choice([16, 32, 64, 128, 256]), "steps": rng.randint(3, 150),
                "nu": rng.uniform(1 / 100, 1 / 20), "dt": rng.uniform(2e-3, 6e-3)}
    if kind == "tangent2d":
        return {"kind": "tangent2d", "n": rng.choice([16, 32, 64, 128, 256]),
                "period": rng.uniform(0.05, 0.5), "nu": rng.uniform(1 / 100, 1 / 20), "dt": 0.005}
    return {"kind": "adjoint3d", "n": rng.choice([16, 32, 64]), "prec": prec, "steps": rng.randint(2, 9),
            "every": rng.randint(1, 5), "nu": max(nu, 1 / 400), "dt": rng.uniform(1e-3, 5e-3)}


# ----------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 1000003)
    return g


def _k3(n):
    g = Grid3D(n)
    K = g.kt
    f = torch.float64
    kx = torch.arange(g.iktx, dtype=f, device="cuda")[None, None, :]
    ky = (torch.arange(g.ikty, dtype=f, device="cuda") - K)[None, :, None]
    kz = (torch.arange(g.iktz, dtype=f, device="cuda") - K)[:, None, None]
    wk = kx * kx + ky * ky + kz * kz
    keep = (kx > 0) | (ky > 0) | ((ky == 0) & (kz > 0))
    keep = keep & (wk <= (K - 0.5) ** 2)
    return kx, ky, kz, wk, keep.to(f), 1.0 / torch.clamp(wk, min=1e-3)


def _curl(k, x):
    kx, ky, kz = k
    return torch.stack([1j * (ky * x[2] - kz * x[1]), 1j * (kz * x[0] - kx * x[2]),
                        1j * (kx * x[1] - ky * x[0])])


def _turbulence3(n, seed, comps):
    """divergence-free vorticity of rms velocity about 1 with a k^-5/3 range and an
    exponential tail at the grid's end (and a density of the same spectrum)"""
    kx, ky, kz, wk, keep, wki = _k3(n)
    g = _gen(seed)
    K = n // 3
    kk = torch.sqrt(torch.clamp(wk, min=1.0))
    amp = keep * kk ** (-11.0 / 6.0) * torch.exp(-3.0 * kk / K)
    z = torch.randn((comps,) + tuple(keep.shape), dtype=torch.complex128, device="cuda", generator=g) * amp
    u = z[:3]
    div = (kx * u[0] + ky * u[1] + kz * u[2]) * wki
    u = torch.stack([u[0] - kx * div, u[1] - ky * div, u[2] - kz * div])
    s = 1.0 / torch.sqrt(2.0 * (u.abs() ** 2).sum())
    w = _curl((kx, ky, kz), u * s)
    return torch.cat([w, z[3:] * s]).contiguous()


def _k2(n, device="cuda"):
    K = n // 3
    kx = torch.arange(K + 1, dtype=torch.float64, device=device)[None, :]
    ky = (torch.arange(2 * K + 1, dtype=torch.float64, device=device) - K)[:, None]
    wk = kx * kx + ky * ky
    keep = ((kx > 0) | (ky > 0)) & (wk <= (K - 0.5) ** 2)
    return kx, ky, wk, keep.to(torch.float64), 1.0 / torch.clamp(wk, min=1e-3)


def _flow2(n, rng):
    """a Kolmogorov-flow state: random phases, vorticity of order one, steep tail"""
    g = Grid2D(n)
    kx, ky = g.wavenumbers()
    kk = np.sqrt(np.maximum(kx * kx + ky * ky, 1.0))
    a = g.mask() * kk ** -1.5 * np.exp(-4.0 * kk / max(g.kt, 8))
    Z = a * np.exp(1j * rng.uniform(-np.pi, np.pi, g.shape))
    return Z * (2.0 / np.sqrt(2 * np.sum(np.abs(Z) ** 2)))


def _sizes(case, seed):
    sizes = [int(s) for s in case["sizes"].split(",")]
    rng = np.random.default_rng(77)  # the ensemble's make-up does not depend on the seed
    mix = [int(s) for s in rng.choice(sizes, case["count"])]
    nu = 1.0 / rng.uniform(20, 100, case["count"])
    r = np.random.default_rng(seed)
    return mix, nu, [_flow2(n, r) for n in mix]


class _DeviceArray:
    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


_LIBS = {}


def _library(flavour):
    if flavour not in _LIBS:
        _LIBS[flavour] = abi.TimestepLibrary(P.dropin_path(flavour), flavour)
    return _LIBS[flavour]


def _upo_periods(case):
    rng = np.random.default_rng(5)
    return rng.uniform(case["tmin"], case["tmax"], case["guesses"])


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("ns3d", "adjoint3d"):
        scheme = SCHEMES[case.get("scheme", "rk4")]
        eng = P.NS3D(case["n"], scheme, precision=case["prec"], nu=case["nu"], ampfor=case.get("ampfor", 0.0),
                     kf=case.get("kf", 4), ri=case.get("ri", 0.0), sc=1.0, theta=case.get("theta", 0.0))
        w = _turbulence3(case["n"], seed, eng.ncomp)
        st = {"case": case, "eng": eng, "w": w}
        if kind == "adjoint3d":
            st["cot"] = _turbulence3(case["n"], seed + 500, eng.ncomp)
        else:
            st["out"] = torch.empty_like(w)
        return st
    if kind == "bous_abi":
        w = _turbulence3(case["n"], seed, 4).cpu()
        host = [w[q].clone().pin_memory() for q in range(4)]
        return {"case": case, "host": host, "comps": [h.numpy() for h in host], "lib": _library("bous3d")}
    if kind == "ns2d_abi":
        return {"case": case, "Z": _flow2(case["n"], np.random.default_rng(seed)), "lib": _library("ns2d")}
    if kind == "batch2d":
        sizes, nu, states = _sizes(case, seed)
        b = P.Batch2D(sizes, precision=case["prec"])
        for i, Z in enumerate(states):
            b.upload(i, Z)
        b.set_params(nu, case["dt"], case["steps"])
        t = "<c8" if case["prec"] == 32 else "<c16"
        views = [torch.as_tensor(_DeviceArray(b.device_state(i), Grid2D(n).shape, t), device="cuda").reshape(-1)
                 for i, n in enumerate(sizes)]
        return {"case": case, "b": b, "views": views}
    rng = np.random.default_rng(seed)
    if kind == "tangent2d":
        u = P.UPO2D(1, case["n"], kmax=8, exact_jv=True)
        u.set_guess(0, _flow2(case["n"], rng), case["period"], nu=case["nu"], dt=case["dt"])
        return {"case": case, "u": u, "q": _flow2(case["n"], rng)}
    u = P.UPO2D(case["guesses"], case["n"], kmax=case["kmax"], exact_jv=True)
    # states near the laminar solution w(0, +-4) = -2 / (16 nu)
    g = Grid2D(case["n"])
    lam = np.zeros(g.shape, np.complex128)
    lam[g.kt + 4, 0] = -2.0 / (16.0 * case["nu"])
    return {"case": case, "u": u, "T": _upo_periods(case),
            "Z": [lam + 0.2 * _flow2(case["n"], rng) for _ in range(case["guesses"])]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ns3d":
        eng, w, out = state["eng"], state["w"], state["out"]
        eng.upload_device([t.data_ptr() for t in w])
        eng.step(case["dt"], case["steps"])
        eng.download_device([t.data_ptr() for t in out])
        # an FP32 run's state is kept as FP32 by its program
        return out if case["prec"] == 64 else out.to(torch.complex64)
    if kind == "adjoint3d":
        w = state["w"].clone().requires_grad_(True)
        end = adjoint.trajectory(w, state["eng"], case["dt"], case["steps"], case["every"])
        loss = (end * state["cot"].conj()).real.sum()
        loss.backward()
        to = torch.complex128 if case["prec"] == 64 else torch.complex64
        return {"end": end.detach().to(to), "grad": w.grad.to(to)}
    if kind == "bous_abi":
        state["lib"].bous3d_inplace(state["comps"], case["n"], case["nu"], case["dt"],
                                    (case["steps"] - 0.5) * case["dt"], ri=case["ri"], theta=case["theta"])
        return state["comps"]
    if kind == "ns2d_abi":
        return state["lib"].ns2d(state["Z"], case["n"], case["nu"], case["dt"], case["steps"])[0]
    if kind == "batch2d":
        state["b"].launch()
        return torch.cat(state["views"])
    if kind == "tangent2d":
        z, q = state["u"].apply(0, 0, state["q"])
        return {"z": z, "jq": q}
    u = state["u"]
    for i, Z in enumerate(state["Z"]):
        u.set_guess(i, Z, float(state["T"][i]), nu=case["nu"], dt=case["dt"])
    u.solve(max_newton=1, tol=1e-10, gmres_tol=case["gmtol"])
    got = [u.get(i) for i in range(case["guesses"])]
    return {"Z": np.stack([g["Z"] for g in got]), "T": np.array([g["T"] for g in got]),
            "residual": np.array([g["residual"] for g in got])}


# ----------------------------------------------------------------- FP64 oracle
class _Exact3:
    """The 3D schemes in plain torch, FP64, on (comps, kz, ky, kx) boxes."""

    def __init__(self, case):
        self.c, self.n = case, case["n"]
        self.scheme = case.get("scheme", "rk4")
        self.kx, self.ky, self.kz, self.wk, self.keep, self.wki = _k3(self.n)
        K, n = self.n // 3, self.n
        self.K = K
        self.pos = torch.tensor([(i - K) % n for i in range(2 * K + 1)], device="cuda")
        # the modes of the kx = 0 plane that the stored half leaves to conjugation
        iy = torch.arange(2 * K + 1, device="cuda")
        self.lower = (iy[None, :] < K) | ((iy[None, :] == K) & (iy[:, None] < K))

    def phys(self, F):
        n, K = self.n, self.K
        p0 = F[..., 0]
        full = torch.where(self.lower, torch.flip(p0, (-1, -2)).conj(), p0)
        one = torch.ones_like(self.lower, dtype=torch.float64)
        one[K, K] = 0.0
        F = torch.cat([(full * one)[..., None], F[..., 1:]], -1)
        A = torch.zeros(F.shape[:-3] + (n, n, n // 2 + 1), dtype=F.dtype, device=F.device)
        A[..., self.pos[:, None, None], self.pos[None, :, None],
          torch.arange(K + 1, device="cuda")[None, None, :]] = F
        return torch.fft.irfftn(A, s=(n, n, n), norm="forward")

    def spec(self, f):
        F = torch.fft.rfftn(f, dim=(-3, -2, -1), norm="forward")
        return F[..., self.pos[:, None, None], self.pos[None, :, None],
                 torch.arange(self.K + 1, device="cuda")[None, None, :]]

    def rhs(self, x):
        """curl F(u x w) (and the density's terms) on the whole box, unmasked"""
        k = (self.kx, self.ky, self.kz)
        u = _curl(k, x[:3]) * self.wki
        pu, pw = self.phys(u), self.phys(x[:3])
        N = _curl(k, self.spec(torch.linalg.cross(pu, pw, dim=0)))
        if self.scheme != "bous":
            return N
        ri, st, ct = self.c["ri"], math.sin(self.c["theta"]), math.cos(self.c["theta"])
        g = torch.stack([1j * a * x[3] for a in k])
        N = N + ri * torch.stack([-(g[1] * st - g[2] * ct), g[0] * st, -g[0] * ct])
        r = -self.spec((pu * self.phys(g)).sum(0)) + u[1] * ct + u[2] * st
        return torch.cat([N, r[None]])

    def forced(self, N):
        a, kf, K = self.c.get("ampfor", 0.0), self.c.get("kf", 4), self.K
        if not a:
            return N
        f = torch.zeros_like(N)
        if self.scheme == "heun":
            f[0, K + kf, K + kf, 0] = a
            f[0, K - kf, K + kf, 0] = -a
        else:
            f[2, K, K + kf, 0] = a
        return N + f

    def run(self, w, steps, last=1.0):
        """`steps` steps of dt, the last of them of `last` times dt (RK4 schemes)"""
        dt, nu, m = self.c["dt"], self.c["nu"], self.keep
        nk = dt * nu * self.wk
        if self.scheme in ("heun", "euler"):
            S = w
            for _ in range(steps):
                if self.scheme == "heun":
                    H = self.forced(self.rhs(S))
                    nu1 = dt / (1 + 0.5 * nk)
                    S = m * ((1 - 0.5 * nk) / (1 + 0.5 * nk) * S + nu1 * H)
                    S = m * (S + 0.5 * nu1 * (self.forced(self.rhs(S)) - H))
                else:
                    H = self.rhs(S)
                    S = S + dt * H
                    S = m * (S + 0.5 * dt * (self.rhs(S) - m * H))
            return S
        S = X = w
        for i in range(steps):
            if i == steps - 1:
                dt, nk = dt * last, nk * last
            N = lambda: self.forced(m * self.rhs(X))  # noqa: E731
            d1 = dt * N()
            X = (1 - 0.25 * nk) / (1 + 0.25 * nk) * (S + 0.5 * d1)
            d2 = dt * N()
            X = (1 - 0.25 * nk) / (1 + 0.25 * nk) * (S + 0.5 * d2)
            d3 = dt * N()
            X = (1 - 0.5 * nk) / (1 + 0.5 * nk) * (S + d3)
            # the last stage's right-hand side is masked with the update
            d4 = dt * N()
            X = m * (((1 - 0.5 * nk) * S + (d1 + d4) / 6 + (d2 + d3) / 3) / (1 + 0.5 * nk))
            div = (self.kx * X[0] + self.ky * X[1] + self.kz * X[2]) * self.wki
            S = torch.cat([torch.stack([X[0] - self.kx * div, X[1] - self.ky * div, X[2] - self.kz * div]), X[3:]])
        return S


class _Exact2:
    """The 2D RK4/CN step and its tangent in plain torch, FP64, on (..., ky, kx) boxes."""

    def __init__(self, n, nu, dt, device="cuda"):
        self.n, self.dt = n, dt
        self.kx, self.ky, self.wk, self.keep, self.wki = _k2(n, device)
        self.nk = dt * nu * self.wk
        K = n // 3
        self.K = K
        self.pos = torch.tensor([(i - K) % n for i in range(2 * K + 1)], device=device)
        self.cols = torch.arange(K + 1, device=device)

    def phys(self, F):
        n, K = self.n, self.K
        F = F.clone()
        F[..., :K, 0] = torch.flip(F[..., K + 1:, 0], (-1,)).conj()
        F[..., K, 0] = 0
        A = torch.zeros(F.shape[:-2] + (n, n // 2 + 1), dtype=F.dtype, device=F.device)
        A[..., self.pos[:, None], self.cols[None, :]] = F
        return torch.fft.irfftn(A, s=(n, n), dim=(-2, -1), norm="forward")

    def fields(self, z):
        z = z * self.keep
        return self.phys(torch.stack([z, 1j * self.ky * self.wki * z, -1j * self.kx * self.wki * z]))

    def div(self, a, b):
        F = torch.fft.rfftn(torch.stack([a, b]), dim=(-2, -1), norm="forward")
        F = F[..., self.pos[:, None], self.cols[None, :]]
        return -1j * (self.kx * F[1] + self.ky * F[0]) * self.keep

    def run(self, z, steps, q=None):
        dt, nk, m, K = self.dt, self.nk, self.keep, self.K
        force = torch.zeros_like(z)
        if K >= 4:
            force[..., K + 4, 0] = -2.0 * m[K + 4, 0]
        z = z * m
        q = None if q is None else q * m

        def rhs(a, b):
            w, u, v = self.fields(a)
            d = dt * (self.div(v * w, u * w) + force)
            if b is None:
                return d, None
            dw, du, dv = self.fields(b)
            return d, dt * self.div(dv * w + v * dw, du * w + u * dw)

        def end(s, ds):
            i = (ds[0] + 2 * ds[1] + 2 * ds[2] + ds[3]) / 6
            return ((1 - 0.5 * nk) * s + i) / (1 + 0.5 * nk) * m

        for _ in range(steps):
            a, b, D, E = z, q, [], []
            for c in (0.5, 0.5, 1.0, 0.0):
                d, e = rhs(a, b)
                D.append(d)
                a = z + c * d
                if q is not None:
                    E.append(e)
                    b = q + c * e
            z = end(z, D)
            if q is not None:
                q = end(q, E)
        return z if q is None else (z, q)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ns3d":
        return _Exact3(case).run(_turbulence3(case["n"], seed, 4 if case["scheme"] == "bous" else 3), case["steps"])
    if kind == "adjoint3d":
        w = _turbulence3(case["n"], seed, 3).requires_grad_(True)
        cot = _turbulence3(case["n"], seed + 500, 3)
        end = w * _k3(case["n"])[4]  # states live on the kept modes
        for _ in range(case["steps"]):  # the gradient is that of steps from each stored state
            end = _Exact3(case).run(end, 1)
        (end * cot.conj()).real.sum().backward()
        return {"end": end.detach(), "grad": w.grad}
    if kind == "bous_abi":
        got = _Exact3(dict(case, scheme="bous")).run(_turbulence3(case["n"], seed, 4), case["steps"],
                                                         last=0.5)
        return [got[q].cpu().numpy() for q in range(4)]
    if kind == "ns2d_abi":
        Z = torch.from_numpy(_flow2(case["n"], np.random.default_rng(seed))).cuda()
        return _Exact2(case["n"], case["nu"], case["dt"]).run(Z, case["steps"]).cpu().numpy()
    if kind == "batch2d":
        sizes, nu, states = _sizes(case, seed)
        out = [None] * len(sizes)
        for n in sorted(set(sizes)):
            at = [i for i, s in enumerate(sizes) if s == n]
            Z = torch.from_numpy(np.stack([states[i] for i in at])).cuda()
            e = _Exact2(n, 1.0, case["dt"])
            e.nk = case["dt"] * torch.from_numpy(nu[at]).cuda()[:, None, None] * e.wk
            for j, z in zip(at, e.run(Z, case["steps"])):
                out[j] = z.reshape(-1)
        return torch.cat(out)
    if kind == "tangent2d":
        rng = np.random.default_rng(seed)
        Z, q = (torch.from_numpy(_flow2(case["n"], rng)).cuda() for _ in range(2))
        steps = int(case["period"] / case["dt"])
        z, j = _Exact2(case["n"], case["nu"], case["period"] / steps).run(Z, steps, q)
        return {"z": z.cpu().numpy(), "jq": j.cpu().numpy()}
    return None


# ----------------------------------------------------------------- work
def _flops3(n, fields):
    return fields * 2.5 * n ** 3 * 3 * math.log2(n)


def _flops2(n, fields):
    return fields * 2.5 * n * n * 2 * math.log2(n)


def work(case):
    """Inputs read once, outputs written once; nominal real-FFT operations, 2.5 N log2 N each."""
    kind = case["kind"]
    n = case.get("n", 0)
    if kind in ("ns3d", "bous_abi"):
        scheme = case.get("scheme", "bous")
        nc, nf = (4, 13) if scheme == "bous" else (3, 9)
        stages = 2 if scheme in ("heun", "euler") else 4
        out = 8 if case.get("prec", 64) == 32 else 16
        return {"bytes": nc * Grid3D(n).nkt * (16 + out), "flops": case["steps"] * stages * _flops3(n, nf)}
    if kind == "adjoint3d":
        # forward once, recomputed once, and per step's adjoint four right-hand sides:
        # nine fields to physical space and six back
        return {"bytes": 3 * Grid3D(n).nkt * 16 * 4, "flops": case["steps"] * 4 * _flops3(n, 9 + 9 + 15)}
    if kind == "ns2d_abi":
        return {"bytes": 2 * Grid2D(n).nkt * 16, "flops": case["steps"] * 4 * _flops2(n, 5)}
    if kind == "batch2d":
        sizes = _mix(case)
        b = 16 if case["prec"] == 64 else 8
        return {"bytes": sum(2 * Grid2D(s).nkt * b for s in sizes),
                "flops": case["steps"] * 4 * sum(_flops2(s, 5) for s in sizes)}
    if kind == "tangent2d":
        return {"bytes": 4 * Grid2D(n).nkt * 16, "flops": int(case["period"] / case["dt"]) * 4 * _flops2(n, 10)}
    steps = sum(int(t / case["dt"]) for t in _upo_periods(case))
    # a Krylov product per guess and dimension, the residual and one trial
    return {"bytes": case["guesses"] * Grid2D(n).nkt * 16 * (2 + 2 * case["kmax"]),
            "flops": steps * 4 * (_flops2(n, 10) * case["kmax"] + 2 * _flops2(n, 5))}


def _mix(case):
    sizes = [int(s) for s in case["sizes"].split(",")]
    return [int(s) for s in np.random.default_rng(77).choice(sizes, case["count"])]
