"""Steps and uploads captured into a CUDA graph and replayed on states the engine
was not told about.  A state with truncated modes must come out as from an engine
that takes the whole box in every pass (device_state), through the same graph: a step
masks those modes, whatever the engine knew of its state when the step was captured."""
import numpy as np
import pytest
import torch

import psgpu_b200 as P
from psgpu_b200.fields import random_vorticity3d

pytestmark = pytest.mark.gpu


def _state(n, nc, truncated, seed):
    g = P.Grid3D(n)
    w = list(random_vorticity3d(n, seed, kmin=0.5, kmax=g.kt - 0.5, solenoidal=True))
    if nc == 4:
        w.append(0.3 * random_vorticity3d(n, seed + 1, kmin=0.5, kmax=g.kt - 0.5)[0])
    w = np.stack(w)
    if truncated:
        rng = np.random.default_rng(seed)
        w = w + 1e-2 * ~g.mask() * (rng.standard_normal(w.shape) + 1j * rng.standard_normal(w.shape))
    return torch.from_numpy(w).cuda()


def _pointers(w):
    return [t.data_ptr() for t in w]


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("n", [32, 64, 128])
@pytest.mark.parametrize("scheme", [P.SCHEME_NS_RK4, P.SCHEME_NS_HEUN, P.SCHEME_BOUS_RK4])
@pytest.mark.parametrize("what", ["step", "first step", "upload"])
def test_replay_on_a_state_with_truncated_modes(monkeypatch, prec, n, scheme, what):
    monkeypatch.setenv("PSG_XPASS_VARIANT", "0")
    monkeypatch.setenv("PSG_PASSA_PACKED", "0")
    out = []
    for whole in (False, True):
        s = torch.cuda.Stream()
        e = P.NS3D(n, scheme, precision=prec, nu=0.01, ampfor=0.1, kf=2, ri=0.5, theta=0.4)
        clean, dirty = _state(n, e.ncomp, False, 3), _state(n, e.ncomp, True, 4)
        src = clean.clone()
        torch.cuda.synchronize()
        e.set_stream(s.cuda_stream)
        if whole:
            e.device_state()
        graph = torch.cuda.CUDAGraph()
        e.upload_device(_pointers(src))
        if what != "first step":
            e.step(2e-3, 1)
        e.sync()
        with torch.cuda.graph(graph, stream=s):
            if what == "upload":
                e.upload_device(_pointers(src))
            else:
                e.step(2e-3, 2)
        with torch.cuda.stream(s):
            if what == "upload":
                e.step(2e-3, 1)
                src.copy_(dirty)
                graph.replay()
                e.step(2e-3, 2)
            else:
                e.upload_device(_pointers(dirty))
                graph.replay()
        e.sync()
        out.append(e.download())
        torch.cuda.synchronize()
        del graph
        e.close()
    mask = P.Grid3D(n).mask()
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.abs(a[~mask]).max() == 0
        np.testing.assert_array_equal(a, b)
