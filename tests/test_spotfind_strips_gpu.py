"""The strong-pixel classifier at the edges of its strips (64 columns of which an extended first pass writes 60;
60, 28, 12 or 4 rows; four rows a step) and over window half-sizes from 0 to the largest, square or not: bit for bit the
oracle, on frames whose values are not whole numbers (so that the order of the window sums shows)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import spotfind as OS

pytestmark = pytest.mark.gpu


def _frames(n, ny, nx, seed):
    rng = np.random.default_rng(seed)
    img = (rng.poisson(0.7, (n, ny, nx)) * rng.uniform(0.8, 1.3, (n, ny, nx))).astype(np.float32)
    for f in range(n):
        for _ in range(max(2, ny * nx // 900)):
            y, x = int(rng.integers(0, ny)), int(rng.integers(0, nx))
            img[f, max(y - 1, 0):y + 2, max(x - 1, 0):x + 2] += np.float32(rng.uniform(4, 5000))
    img[:, :, nx // 3] = -1.0
    img[:, ny // 2, :] = -2.0
    return img


def _check(img, **kw):
    from xpg_b200.spotfind import make_finder
    want_s, want_m = OS.find(img, 1.3, **kw)
    s, m = make_finder(**kw)(torch.from_numpy(img).cuda(), 1.3)
    assert s.dtype == torch.bool
    assert np.array_equal(s.cpu().numpy(), want_s)
    assert np.array_equal(m.cpu().numpy(), want_m)


@pytest.mark.parametrize("ny,nx", [(1, 1), (3, 5), (4, 59), (5, 60), (12, 61), (13, 63), (28, 64), (29, 65), (60, 120),
                                   (61, 121), (63, 128), (65, 129), (240, 3001)])
@pytest.mark.parametrize("extended", [False, True])
def test_strip_edges(ny, nx, extended):
    _check(_frames(2, ny, nx, 7 * ny + nx), extended=extended)


@pytest.mark.parametrize("nbx,nby", [(0, 0), (1, 1), (2, 2), (4, 4), (5, 5), (8, 8), (0, 3), (3, 1), (8, 2), (2, 8)])
@pytest.mark.parametrize("extended", [False, True])
def test_window_sizes(nbx, nby, extended):
    _check(_frames(1, 70, 300, 31 * nbx + nby), nbx=nbx, nby=nby, extended=extended)


def test_long_strips():
    """Enough strips for the longest march (60 rows) and its remainder."""
    _check(_frames(30, 201, 1100, 5))
