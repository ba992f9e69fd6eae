"""The linearised right-hand sides' fused products (nine fields for the adjoint,
twelve for the tangent, through the five passes once) at every grid size's tile
shapes: the tangent and the adjoint are transposes of each other in the real inner
product of the stored coefficients, the tangent is linear, and FP32 follows FP64.

Tolerances: the products are sums of N^3 terms scaled by 1/N^3 whose transforms
err by a few eps log2 N^3; relative to the norms that enter, 1e-13 (FP64) and 2e-5
(FP32, with the inner products themselves accumulated in FP64) leave a factor of
ten."""
import numpy as np
import pytest
import torch

import psgpu_b200 as P

pytestmark = pytest.mark.gpu


def _field(n, seed):
    g = P.Grid3D(n)
    rng = np.random.default_rng(seed)
    kx, ky, kz = g.wavenumbers()
    a = g.mask() / (1.0 + kx * kx + ky * ky + kz * kz)
    z = a * (rng.standard_normal((3,) + g.shape) + 1j * rng.standard_normal((3,) + g.shape))
    return torch.from_numpy(z).cuda()


def _dot(a, b):
    return float((a.conj() * b).real.sum())


@pytest.mark.parametrize("n", [16, 32, 64, 128])
def test_tangent_and_adjoint_products(n):
    z, x, l = (_field(n, s) for s in (1, 2, 3))
    out = {}
    for prec, tol in ((64, 1e-13), (32, 2e-5)):
        e = P.NS3D(n, P.SCHEME_NS_RK4, precision=prec, nu=0.01)
        e.upload_device([t.data_ptr() for t in z])
        jx = e.linear(P.NS3D.LIN_TANGENT_RHS, x)
        jl = e.linear(P.NS3D.LIN_ADJOINT_RHS, l)
        j2 = e.linear(P.NS3D.LIN_TANGENT_RHS, 2.0 * x + l)
        jlx = e.linear(P.NS3D.LIN_TANGENT_RHS, l)
        e.sync()
        size = float(torch.linalg.norm(jx) * torch.linalg.norm(l) + torch.linalg.norm(x) * torch.linalg.norm(jl))
        assert abs(_dot(jx, l) - _dot(x, jl)) < tol * size
        assert float(torch.linalg.norm(j2 - 2.0 * jx - jlx)) < 10 * tol * float(torch.linalg.norm(j2))
        out[prec] = (jx, jl)
        e.close()
    for a, b in zip(out[32], out[64]):
        assert float(torch.linalg.norm(a - b)) < 2e-5 * float(torch.linalg.norm(b))
