"""The on-chip 2D integrator (one instance per thread-block cluster) at every
cluster size its dispatch picks, and the FP64 global-memory kernel of large
batches, against the FP64 oracle: the counts put each grid at the edges of the
dispatch (one run on the most blocks, the last count that still gets several, the
first that gets one block or the global kernel), with ragged step counts, a run of
no steps among them.

Tolerance: a step adds a few roundings of the state to transforms whose error is
a few eps log2 N; three steps stay below 1e-12 (FP64, eps 1.1e-16) and 2e-6
(FP32, eps 6e-8) of the largest mode.
"""
import numpy as np
import pytest

import psgpu_b200 as P
from oracle import pyoracle as O
from psgpu_b200.fields import kolmogorov_ic2d

pytestmark = pytest.mark.gpu

TOL = {64: 1e-12, 32: 2e-6}


def _check(sizes, prec):
    rng = np.random.default_rng(len(sizes))
    m = len(sizes)
    nu = 1.0 / rng.uniform(20, 100, m)
    ns = (np.arange(m) % 3 + 1).astype(np.int32)
    if m > 2:
        ns[1] = 0
    ic = {n: kolmogorov_ic2d(n, 50 + n) for n in set(sizes)}
    b = P.Batch2D(sizes, precision=prec)
    for i, n in enumerate(sizes):
        b.upload(i, ic[n])
    b.run(nu, 0.005, ns)
    for i in sorted({0, 1 % m, m // 2, m - 1}):
        ref = O.ns2d_timestep(ic[sizes[i]], sizes[i], nu[i], 0.005, int(ns[i]))[0] if ns[i] else ic[sizes[i]]
        err = np.max(np.abs(b.download(i) - ref)) / np.max(np.abs(ref))
        assert err < TOL[prec], (prec, sizes[i], m, i, err)
    b.close()


@pytest.mark.parametrize("prec,n,count", [
    (64, 16, 1), (64, 32, 3), (64, 64, 1), (64, 64, 15), (64, 64, 16), (64, 64, 66), (64, 64, 67), (64, 128, 1), (64, 128, 7),
    (64, 128, 15), (64, 128, 16), (64, 128, 132), (64, 128, 133), (64, 256, 1), (64, 256, 8), (64, 256, 97),
    (32, 16, 2), (32, 32, 1), (32, 64, 1), (32, 64, 66), (32, 64, 67), (32, 128, 15), (32, 128, 16), (32, 128, 34),
    (32, 128, 75), (32, 256, 1), (32, 256, 7), (32, 256, 8)])
def test_one_size_matches_oracle(prec, n, count):
    _check([n] * count, prec)


@pytest.mark.parametrize("prec", [64, 32])
def test_mixed_sizes_match_oracle(prec):
    _check([256, 16, 128, 64, 32, 128, 256, 64], prec)


def test_large_mixed_fp64_batch_matches_oracle():
    """128^2 through the global-memory kernel beside on-chip sizes"""
    _check([128] * 133 + [256, 64, 32], 64)
