"""The plane kernel (passes B, C and D in one launch, up to 64^3) against the
separate passes it stands for, which an engine created under PSG_PLANE=0 takes at
every size: whole steps with their kept physical fields, and the linearised step's
right-hand sides, whose buffers follow the same choice.

Both do the same transforms, with the products in another order: a step or a
right-hand side differs by a few roundings, below 1e-13 (FP64) and 2e-6 (FP32) of the
largest value."""
import numpy as np
import pytest
import torch

import psgpu_b200 as P
from psgpu_b200.fields import random_vorticity3d

pytestmark = pytest.mark.gpu

TOL = {64: 1e-13, 32: 2e-6}


def _engines(monkeypatch, n, scheme, prec, **kw):
    out = []
    for plane in ("1", "0"):
        monkeypatch.setenv("PSG_PLANE", plane)
        monkeypatch.setenv("PSG_PASSA_PACKED", "0")
        out.append(P.NS3D(n, scheme, precision=prec, nu=0.01, **kw))
    return out


def _state(n, nc):
    w = list(random_vorticity3d(n, 5, kmin=0.5, kmax=n // 3 - 0.5, solenoidal=True))
    if nc == 4:
        w.append(0.3 * random_vorticity3d(n, 6, kmin=0.5, kmax=n // 3 - 0.5)[0])
    return w


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("n", [16, 32, 64])
@pytest.mark.parametrize("scheme", [P.SCHEME_NS_RK4, P.SCHEME_NS_HEUN, P.SCHEME_EULER_HEUN, P.SCHEME_BOUS_RK4])
def test_steps(monkeypatch, prec, n, scheme):
    heun = scheme in (P.SCHEME_NS_HEUN, P.SCHEME_EULER_HEUN)
    got = []
    for e in _engines(monkeypatch, n, scheme, prec, ampfor=0.1, kf=2, ri=0.5, theta=0.4):
        e.upload(*_state(n, e.ncomp))
        before = e.launches
        e.step(2e-3, 2, dump_last=heun)
        launches = e.launches - before
        got.append((e.download(), e.physical() if heun else None, launches))
        e.close()
    (a, pa, la), (b, pb, lb) = got
    # three launches a right-hand side against five, but for 64^3 FP32 Navier-Stokes and
    # the right-hand side whose fields are kept at 64^3
    assert lb == 5 * (4 if heun else 8)
    assert (la < lb) == (n < 64 or prec == 64 or scheme == P.SCHEME_BOUS_RK4)
    for x, y in zip(a, b):
        assert _rel(x, y) < TOL[prec]
    if heun:
        assert _rel(pa, pb) < TOL[prec]


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("n", [16, 32, 64])
@pytest.mark.parametrize("scheme", [P.SCHEME_NS_RK4, P.SCHEME_BOUS_RK4])
def test_linearised(monkeypatch, prec, n, scheme):
    got = []
    for e in _engines(monkeypatch, n, scheme, prec, ri=0.5, theta=0.4):
        w = torch.from_numpy(np.stack(_state(n, e.ncomp))).cuda()
        x = torch.roll(w, 1, 0).contiguous()
        e.upload_device([t.data_ptr() for t in w])
        out = [e.linear(m, x, 2e-3) for m in (P.NS3D.LIN_TANGENT_RHS, P.NS3D.LIN_ADJOINT_RHS,
                                              P.NS3D.LIN_TANGENT_STEP, P.NS3D.LIN_ADJOINT_STEP)]
        e.sync()
        got.append([t.cpu().numpy() for t in out])
        e.close()
    for x, y in zip(*got):
        assert np.isfinite(y).all()
        assert _rel(x, y) < 10 * TOL[prec]  # four right-hand sides a step
