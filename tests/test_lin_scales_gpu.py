"""The linearised right-hand sides at any ratio of the perturbation to the state: no
transform line holds a field of each, so that a perturbation scaled by a power of two
gives a result scaled by it, bit for bit; and an FP32 gradient's error does not grow by
rounding of the state's size (an adjoint step's right-hand sides take dt times the
adjoint): through 24 adjoint steps of 2^-8 it stays within sqrt(24) roundings of the
adjoint's own, 0.5 eps each of four additions a step, 5e-7 of its norm."""
import numpy as np
import pytest
import torch

import psgpu_b200 as P

pytestmark = pytest.mark.gpu


def _fields(n, nc, seed):
    g = P.Grid3D(n)
    kx, ky, kz = g.wavenumbers()
    kk = np.sqrt(np.maximum(kx * kx + ky * ky + kz * kz, 1.0))
    rng = np.random.default_rng(seed)
    a = g.mask() * kk ** (-11 / 6) * np.exp(-3.0 * kk / g.kt)
    z = a * (rng.standard_normal((nc,) + g.shape) + 1j * rng.standard_normal((nc,) + g.shape))
    return torch.from_numpy(z.astype(np.complex64).astype(np.complex128)).cuda()


@pytest.mark.parametrize("plane", ["1", "0"])
@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("n", [16, 32, 64, 128])
@pytest.mark.parametrize("scheme", [P.SCHEME_NS_RK4, P.SCHEME_BOUS_RK4])
def test_scaled_perturbation(monkeypatch, plane, prec, n, scheme):
    if n == 128 and plane == "1":
        pytest.skip("no plane kernel at this size")
    monkeypatch.setenv("PSG_PLANE", plane)
    e = P.NS3D(n, scheme, precision=prec, nu=0.01, ri=0.5, theta=0.4)
    z, x = (_fields(n, e.ncomp, s) for s in (1, 2))
    e.upload_device([t.data_ptr() for t in z])
    modes = [P.NS3D.LIN_ADJOINT_RHS]
    if scheme == P.SCHEME_NS_RK4:  # the Boussinesq tangent is a central difference about z
        modes.append(P.NS3D.LIN_TANGENT_RHS)
    for mode in modes:
        one = e.linear(mode, x)
        for p in (-20, 12):
            assert torch.equal(e.linear(mode, x * 2.0 ** p), one * 2.0 ** p), (mode, p)
    e.sync()
    e.close()


@pytest.mark.parametrize("n", [32, 64])
def test_fp32_adjoint_steps(n):
    z, x = (_fields(n, 3, s) for s in (3, 4))
    out = {}
    for prec in (64, 32):
        e = P.NS3D(n, P.SCHEME_NS_RK4, precision=prec, nu=2.0 ** -7)
        lam = x.clone()
        for _ in range(24):
            e.upload_device([t.data_ptr() for t in z])
            lam = e.linear(P.NS3D.LIN_ADJOINT_STEP, lam, 2.0 ** -8)
        e.sync()
        out[prec] = lam
        e.close()
    err = float(torch.linalg.norm(out[32] - out[64]) / torch.linalg.norm(out[64]))
    assert err < 5e-7, err
