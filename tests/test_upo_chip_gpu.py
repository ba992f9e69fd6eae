"""The UPO search's integrations on the on-chip kernels (64^2 to 256^2) against the
oracle, at the shapes their dispatch picks and at each that is built.

* dz/dt and Phi_T (FP64) against the oracle: a few eps log2 N per step, 1e-12 of the
  largest mode; the exact tangent against central differences of the oracle's step,
  whose truncation O(eps^2) = 1e-10 and rounding 1e-16 / eps = 1e-11 leave 1e-7 ample;
* the FP32 tangent against the FP64 one: eps 6e-8 through 3 log2 N butterflies and
  the sums of four stages a step, over four steps, 1e-5;
* every cluster size that is built gives the same integration up to the order in
  which the compiler contracts products into sums: 1e-13 (FP64), 1e-6 (FP32).
"""
import numpy as np
import pytest

import psgpu_b200 as P
from oracle import pyoracle as O
from psgpu_b200.fields import Grid2D, kolmogorov_ic2d
from tests.golden_cases import relerr

pytestmark = pytest.mark.gpu

NU, DT, STEPS = 1 / 40, 0.005, 4


def _direction(n, seed):
    g = Grid2D(n)
    rng = np.random.default_rng(seed)
    kx, ky = g.wavenumbers()
    q = (rng.standard_normal(g.shape) + 1j * rng.standard_normal(g.shape)) * g.mask() / (1.0 + kx * kx + ky * ky)
    return q / np.sqrt(np.sum(np.abs(q) ** 2))


def _search(n, guesses=1, prec=64, T=STEPS * DT):
    u = P.UPO2D(guesses, n, kmax=4, jv_precision=prec)
    Z = kolmogorov_ic2d(n, 5) * 3.0
    for i in range(guesses):
        u.set_guess(i, Z, T=T, nu=NU, dt=DT)
    return u, Z


@pytest.mark.parametrize("n", [64, 128, 256])
def test_timederiv_matches_oracle(n):
    u, Z = _search(n)
    assert u.shape(2)[0] > 0
    d, _ = u.apply(0, 2)
    assert relerr(d, O.ns2d_timederiv(Z, n, NU)) < 1e-12


@pytest.mark.parametrize("n", [64, 128, 256])
def test_phi_matches_oracle(n):
    u, Z = _search(n)
    phi, _ = u.apply(0, 1)
    assert relerr(phi, O.ns2d_timestep(Z, n, NU, DT, STEPS)[0]) < 1e-12


@pytest.mark.parametrize("n", [64, 128, 256])
def test_tangent_matches_central_differences(n):
    q = _direction(n, 6)
    u, Z = _search(n)
    assert (u.shape(0)[0] > 0) == (n < 256)
    phi, jq = u.apply(0, 0, q)
    assert relerr(phi, O.ns2d_timestep(Z, n, NU, DT, STEPS)[0]) < 1e-12
    eps = 1e-5
    zp, zm = (O.ns2d_timestep(Z + s * eps * q, n, NU, DT, STEPS)[0] for s in (1, -1))
    assert relerr(jq, (zp - zm) / (2 * eps)) < 1e-7
    assert relerr(u.apply(0, 0, 2.0 * q)[1], 2.0 * jq) < 1e-14


@pytest.mark.parametrize("n", [64, 128, 256])
def test_fp32_tangent_follows_fp64(n):
    q = _direction(n, 7)
    got = []
    for prec in (64, 32):
        u, _ = _search(n, prec=prec)
        assert prec == 64 or u.shape(0, 32)[0] > 0
        got.append(u.apply(0, 0, q))
    for a, b in zip(got[1], got[0]):
        assert relerr(a, b) < 1e-5


@pytest.mark.parametrize("n,prec,clusters", [(64, 64, (1, 4, 8)), (128, 64, (8, 16)), (64, 32, (1, 4, 8)),
                                             (128, 32, (4, 8))])
def test_built_clusters_agree(monkeypatch, n, prec, clusters):
    q = _direction(n, 8)
    out = []
    for cs in clusters:
        monkeypatch.setenv("PSG_UPO_CLUSTER", str(cs))
        u, _ = _search(n, prec=prec)
        assert u.shape(0, prec)[0] == cs
        out.append(u.apply(0, 0, q) + u.apply(0, 1)[:1] + u.apply(0, 2)[:1])
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            assert relerr(a, b) < {64: 1e-13, 32: 1e-6}[prec]


def test_shape_follows_the_batch():
    """64^2 FP64 tangents on a B200: the most blocks for a few, one block each once
    clusters would take two waves (us a step of 99: 66 on one block, 81 on four, 91 on
    eight)"""
    u, _ = _search(64)
    assert [u.shape(0, 64, m)[0] for m in (1, 15, 99, 148)] == [8, 8, 1, 1]


def test_large_batch_matches_a_small_one():
    """one Newton iteration of 99 guesses (one block each) and of the same three alone
    (a cluster each); GMRES and the hookstep carry rounding of 1e-13 through a few
    Krylov products, 1e-8 of the state"""
    n = 64
    rng = np.random.default_rng(3)
    periods = rng.uniform(0.02, 0.06, 99)
    starts = {i: kolmogorov_ic2d(n, 100 + i) * 2.0 for i in range(99)}
    res = {}
    for who in (range(99), (0, 50, 98)):
        u = P.UPO2D(len(who), n, kmax=4)
        for j, i in enumerate(who):
            u.set_guess(j, starts[i], T=float(periods[i]), nu=NU, dt=DT)
        u.solve(max_newton=1, tol=1e-10)
        res[len(who)] = {i: u.get(j) for j, i in enumerate(who)}
        u.close()
    for i, b in res[3].items():
        a = res[99][i]
        assert relerr(a["Z"], b["Z"]) < 1e-8 and a["gmres"] == b["gmres"]
        assert a["residual"] == pytest.approx(b["residual"], rel=1e-6)
