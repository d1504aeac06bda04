"""The classifier's scratch grows with the frames of a call, so that scratch for a batch serves a shorter one."""
from __future__ import annotations

import pytest

from xpg_b200 import native as N


@pytest.mark.parametrize("ny,nx", [(1, 1), (260, 256), (1030, 1065), (500, 2000), (4148, 4362)])
def test_workspace_grows_with_the_frames(ny, nx):
    lib = N.load()
    sizes = [int(lib.xi_spot_workspace(n, ny, nx)) for n in range(0, 40)]
    assert sizes[0] == 0 and all(a <= b for a, b in zip(sizes, sizes[1:]))
