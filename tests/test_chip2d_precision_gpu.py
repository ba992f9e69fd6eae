"""The FP32 on-chip 2D integrator errs no more than the one-block kernel it took the
place of (which the allocation-free step still runs): RMS distance from the FP64
integration over 16 runs of 20 steps, of the FP32 states as stored.  Both are the same
arithmetic up to contraction, so 2% more would be another algorithm's error."""
import ctypes as C

import numpy as np
import pytest
import torch

import psgpu_b200 as P
from psgpu_b200.fields import Grid2D

pytestmark = pytest.mark.gpu

DT, STEPS, RUNS = float(np.float32(0.005)), 20, 16


def _flow(n, rng):
    g = Grid2D(n)
    kx, ky = g.wavenumbers()
    kk = np.sqrt(np.maximum(kx * kx + ky * ky, 1.0))
    a = g.mask() * kk ** -1.5 * np.exp(-4.0 * kk / max(g.kt, 8))
    Z = a * np.exp(1j * rng.uniform(-np.pi, np.pi, g.shape))
    return (Z * (2.0 / np.sqrt(2 * np.sum(np.abs(Z) ** 2)))).astype(np.complex64)


def _batch(Z, n, prec, nu):
    b = P.Batch2D([n] * RUNS, precision=prec)
    for i in range(RUNS):
        b.upload(i, Z[i].astype(np.complex128))
    b.run(nu, DT, np.full(RUNS, STEPS, np.int32))
    out = np.stack([b.download(i) for i in range(RUNS)])
    b.close()
    return out


def _rms(a, b):
    return float(np.sqrt((np.abs(a - b) ** 2).sum() / (np.abs(b) ** 2).sum()))


@pytest.mark.parametrize("n", [16, 32, 64, 128])
def test_fp32_error(n):
    rng = np.random.default_rng(n)
    Z = [_flow(n, rng) for _ in range(RUNS)]
    nu = (1.0 / rng.uniform(20, 100, RUNS)).astype(np.float32).astype(np.float64)
    ref = _batch(Z, n, 64, nu)
    chip = _batch(Z, n, 32, nu).astype(np.complex64)
    one = []
    for i in range(RUNS):
        d = torch.from_numpy(Z[i]).cuda()
        assert P.lib().psg_ns2d_step_noalloc(n, 32, nu[i], DT, STEPS, C.c_void_p(d.data_ptr()),
                                             C.c_void_p(d.data_ptr()), None) == 0
        torch.cuda.synchronize()
        one.append(d.cpu().numpy())
    assert _rms(chip, ref) <= 1.02 * _rms(np.stack(one), ref)
