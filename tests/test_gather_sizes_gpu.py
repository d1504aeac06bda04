"""The gather's launches (half the threads when the largest box is small, float frames eight at a time in large boxes, a
largest box that is not known) on rows of several shapes, binned and super-pixel rows among them, over two wedges with
an excluded frame and boxes across the frame's border, bit for bit the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import gather as OG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("known", [True, False])
@pytest.mark.parametrize("is_float", [False, True])
@pytest.mark.parametrize("sides", [(3, 5, 9), (11,), (9, 17), (17, 19), (5, 31), (73,)])
def test_gather_matches_oracle(sides, is_float, known):
    from xpg_b200 import device as D
    rng = np.random.default_rng(sum(sides))
    nf, ny, nx, n = 31, 83, 90, 24
    raw = rng.poisson(3.0, (nf, ny, nx)).astype(np.uint32)
    raw[rng.random(raw.shape) < 0.01] = 0xFFFFFFFF
    raw[rng.random(raw.shape) < 0.01] = 5000
    mask = rng.random((ny, nx)) > 0.02
    excluded = 7
    prep = [OG.prepare_frame(r, 1000, 0, mask) for r in raw]
    bx = rng.choice(sides, n).astype(np.int64)
    Dz = rng.choice((1, 3, 5, 9, 17), n).astype(np.int64)
    fb = np.where(np.arange(n) % 6 == 5, 2, 1)
    pxs = np.where(np.arange(n) % 5 == 4, 2, 1)
    iz0, iy0, ix0 = rng.integers(-3, nf, n), rng.integers(-6, ny - 2, n), rng.integers(-6, nx - 2, n)
    z = np.zeros(n, np.float32)
    rows = D.RowSet(S=np.zeros((n, 3), np.float32), phi=z, ix0=ix0, iy0=iy0, iz0=iz0, fb=fb.astype(np.float32),
                    region=z.astype(np.int32), has_p=z, pS=np.zeros((n, 3), np.float32), pphi=z, pxs=pxs, Dz=Dz, bx=bx,
                    nb={k: np.zeros((n, 1), np.float32) for k in ("x", "y", "z", "sx", "sz")})
    g = D.GatherRows(rows, ix0, iy0, iz0, fb, pxs)
    assert g.s.max_bx == bx.max()
    if not known:
        g.s.max_bx = 0
    arena = torch.zeros(rows.n_vox, device="cuda")
    cnt = torch.zeros(max(g.n_cnt, 1), dtype=torch.int32, device="cuda")
    order = torch.as_tensor(rng.permutation(n).astype(np.int32)).cuda()
    mask_t = torch.as_tensor(mask.astype(np.uint8)).cuda()
    for a, b in ((0, 13), (13, nf)):
        data = np.stack(prep[a:b]) if is_float else raw[a:b].view(np.int32)
        ok = torch.as_tensor((np.arange(a, b) != excluded).astype(np.uint8)).cuda()
        data = torch.as_tensor(np.ascontiguousarray(data)).cuda()
        D.gather(D.frames_struct(data, a, 1000, 0, None if is_float else mask_t, ok), g, order, arena, cnt)
    if g.any_binned:
        D.decode_bins(g, arena, cnt)
    got = arena.cpu().numpy()
    ids = [f for f in range(nf) if f != excluded]
    at = {s: [OG.superpixel_frame(p, s) if s > 1 else p for p in prep] for s in (1, 2)}
    for j in range(n):
        want = OG.gather_shoebox(at[int(pxs[j])], ids, int(iz0[j]), int(fb[j]), int(Dz[j]), int(bx[j]), int(iy0[j]), int(ix0[j]))
        box = got[rows.sb_off[j]:rows.sb_off[j] + want.size].reshape(want.shape)
        assert np.array_equal(box - np.float32(3.0), want), (j, bx[j], Dz[j], fb[j], pxs[j])
