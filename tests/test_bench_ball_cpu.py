"""bench.py's bytes within the ball of kept modes: every kept mode is counted, and the
lines and modes are those of the passes' tiles (8 kx columns)."""
import numpy as np
import pytest

import bench
from psgpu_b200.fields import Grid3D


@pytest.mark.parametrize("n", [16, 32, 64, 128])
def test_ball_covers_the_kept_modes(n):
    K = n // 3
    lines, modes = bench.ball_lines(n, w=1)
    m = Grid3D(n).mask()  # (kz, ky, kx)
    half = (K + 1) * (2 * K + 1) ** 2
    # with one column a tile the ball is the mask and, on kx = 0, its conjugate half
    kx0 = int(m[:, :, 0].sum())
    assert modes == int(m.sum()) + kx0 + 1
    wide = bench.ball_lines(n)
    assert lines <= wide[0] <= (K + 1) * (2 * K + 1) and modes <= wide[1] < half


def test_trimmed_bytes_256():
    K, X, Y = 85, 86, 171
    kx, k = np.arange(X) // 8 * 8, np.arange(-K, K + 1)
    inside = kx[:, None, None] ** 2 + k[:, None] ** 2 + k ** 2 <= (K - 0.5) ** 2
    lines, modes = int(inside.any(-1).sum()), int(inside.sum())
    assert bench.ball_lines(256) == (lines, modes)
    whole, ball = bench.algorithmic_bytes(256, 8), bench.algorithmic_bytes(256, 8, ball=True)
    assert ball[2] == whole[2]
    assert ball[4] * X * Y == whole[4] * lines
    assert bench.stage_bytes(256, 0, ball=True) * X * Y * Y == bench.stage_bytes(256, 0) * modes
