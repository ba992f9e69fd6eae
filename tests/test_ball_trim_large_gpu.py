"""The trimmed passes against the whole box at 256^3, where trimming matters most:
test_ball_trim_gpu's comparison, bit for bit, for a masked and a truncated state."""
import pytest

import psgpu_b200 as P
from tests import test_ball_trim_gpu as trim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,scheme,kf,truncated", [
    (32, P.SCHEME_NS_RK4, 2, False), (32, P.SCHEME_NS_RK4, "out", True), (64, P.SCHEME_NS_HEUN, 2, True),
    (32, P.SCHEME_BOUS_RK4, 2, False)])
def test_256(prec, scheme, kf, truncated, monkeypatch):
    trim.test_trimmed_passes_match_the_whole_box(prec, 256, scheme, kf, truncated, monkeypatch)
