"""The strong-pixel classifier by its two routes, strips (many or large frames) and tiles (few small ones), on the same
shapes, and on values that the strips' bounds must leave to the exact tests: infinities, NaN, gains far from one and
negative thresholds. Bit for bit the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import spotfind as OS
from test_spotfind_strips_gpu import _frames

pytestmark = pytest.mark.gpu

STRIPS = 1776                                              # strips of 60 columns and 12 rows that every window marches by


def _check(img, gain=1.3, **kw):
    from xpg_b200.spotfind import make_finder
    with np.errstate(all="ignore"):
        want_s, want_m = OS.find(img, gain, **kw)
    s, m = make_finder(**kw)(torch.from_numpy(img).cuda(), gain)
    assert np.array_equal(s.cpu().numpy(), want_s)
    assert np.array_equal(m.cpu().numpy(), want_m, equal_nan=True)


def _many(ny, nx, seed):
    n = -(-STRIPS // (-(-nx // 60) * -(-ny // 12)))
    few = _frames(min(n, 12), ny, nx, seed)
    return np.ascontiguousarray(few[np.arange(n) % len(few)])


@pytest.mark.parametrize("ny,nx", [(1, 1), (3, 5), (4, 59), (5, 60), (12, 61), (13, 63), (28, 64), (29, 65), (61, 121),
                                   (65, 129)])
@pytest.mark.parametrize("extended", [False, True])
def test_strip_edges_of_many_frames(ny, nx, extended):
    _check(_many(ny, nx, 3 * ny + nx), extended=extended)


@pytest.mark.parametrize("nbx,nby", [(0, 0), (1, 1), (2, 2), (4, 4), (6, 6), (8, 8), (0, 3), (8, 2), (2, 8)])
@pytest.mark.parametrize("extended", [False, True])
def test_strip_windows_of_many_frames(nbx, nby, extended):
    _check(_many(61, 130, 31 * nbx + nby), nbx=nbx, nby=nby, extended=extended)


@pytest.mark.parametrize("gain,kw", [(1.3, {}), (0.0, {}), (1e6, {}), (1e-4, {}), (1.0, dict(signal_pixel=-1.0)),
                                     (1.0, dict(background_pixel=-0.5)), (1.0, dict(background_pixel=0.0, min_local=40)),
                                     (2.0, dict(nbx=5, nby=1))])
@pytest.mark.parametrize("extended", [False, True])
@pytest.mark.parametrize("many", [False, True])
def test_values_that_the_bounds_leave_open(many, extended, gain, kw):
    img = _many(61, 130, 11) if many else _frames(2, 61, 130, 11)
    rng = np.random.default_rng(5)
    for f in range(len(img)):
        for v in (np.nan, np.inf, 1.0e18, 1.0e-40):
            if f % 4 and np.isinf(v):
                continue                                   # (an infinite pixel blanks its windows)
            y, x = rng.integers(0, 61, 2), rng.integers(0, 130, 2)
            img[f, y, x] = np.float32(v)
    _check(img, gain, extended=extended, **kw)
