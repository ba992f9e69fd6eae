"""The five separate passes at small grids.  Up to 64^3 a step takes the plane kernel
in place of passes B, C and D; 128^3 and 256^3 take the passes.  Under PSG_PLANE=0
every grid does, so that the comparisons that run at small grids (the reference's
golden steps, the x-pass schedules, launch chaining, trimming) reach them in every
precision and scheme: the tests of those files, in a process of their own, with the
tolerances they state."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("tests", [
    ["tests/test_parity_gpu.py", "-k", "golden or ns3d or masked"], ["tests/test_xpass_variants_gpu.py"],
    ["tests/test_pdl_gpu.py"], ["tests/test_ball_trim_gpu.py", "-k", "not 128"], ["tests/test_lin_products_gpu.py"],
    ["tests/test_passa_packed_gpu.py"]], ids=lambda t: os.path.basename(t[0])[5:-7])
def test_under_separate_passes(tests):
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider", *tests],
                       cwd=ROOT, env=dict(os.environ, PSG_PLANE="0"), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-1000:]
    assert " passed" in r.stdout
