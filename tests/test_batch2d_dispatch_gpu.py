"""Batches of the 2D engine beside each other and at the edges of what holds them."""
import numpy as np
import pytest

import psgpu_b200 as P
from oracle import pyoracle as O
from psgpu_b200.fields import kolmogorov_ic2d

pytestmark = pytest.mark.gpu


def _batch(n, count, prec=64, nu=0.02):
    b = P.Batch2D([n] * count, precision=prec)
    for i in range(count):
        b.upload(i, kolmogorov_ic2d(n, 50 + n))
    b.set_params(np.full(count, nu), 0.005, np.ones(count, np.int32))
    return b


def _error(b, i, n, nu=0.02):
    ref = O.ns2d_timestep(kolmogorov_ic2d(n, 50 + n), n, nu, 0.005, 1)[0]
    return np.max(np.abs(b.download(i) - ref)) / np.max(np.abs(ref))


def test_two_large_fp64_batches_alive():
    """Both run the global-memory kernel, whose shared-memory limit belongs to the
    process: the second batch needs less of it than the first, which launches (and,
    in the other order of creation, autotunes) after the second was created.
    Tolerance as one FP64 step's, a few eps log2 N of the largest mode."""
    a = _batch(128, 133)
    b = _batch(256, 97)
    a.launch()
    b.launch()
    assert _error(a, 132, 128) < 1e-12 and _error(b, 96, 256) < 1e-12
    b.close()
    c = _batch(128, 133)
    d = _batch(256, 97)
    c.autotune()
    c.launch()
    assert _error(c, 0, 128) < 1e-12
    for x in (a, c, d):
        x.close()


@pytest.mark.parametrize("prec,n,most", [(64, 256, 8), (64, 128, 2), (32, 256, 4), (64, 64, 2), (32, 64, 4), (32, 128, 2)])
def test_no_room_for_the_cluster(monkeypatch, prec, n, most):
    """PSG_2D_CLUSTER bounds the cluster, as a part of a GPU does: grids that need
    more blocks run on the global-memory kernel, beside sizes that fit.  Three steps,
    tolerance as for the on-chip kernels."""
    monkeypatch.setenv("PSG_2D_CLUSTER", str(most))
    sizes = [n, 32, n]
    b = P.Batch2D(sizes, precision=prec)
    for i, m in enumerate(sizes):
        b.upload(i, kolmogorov_ic2d(m, 50 + m))
    b.run(np.full(3, 0.02), 0.005, np.full(3, 3, np.int32))
    for i, m in enumerate(sizes):
        ref = O.ns2d_timestep(kolmogorov_ic2d(m, 50 + m), m, 0.02, 0.005, 3)[0]
        assert np.max(np.abs(b.download(i) - ref)) < {64: 1e-12, 32: 2e-6}[prec] * np.max(np.abs(ref))
    b.close()
