"""Pass 1 and pass 2 at the shapes where their loops end unevenly (frame batches of eight, nine and seventeen, runs of
nine, boxes of fewer or slightly more pixels than a CTA has threads), with the box staged or not, both CTA widths and
a fit list that holds all, some or none of the fitted voxels, against the oracle: masks, counts and per-pixel terms bit
for bit, sums within 1e-5 (pass 1) and 2e-6 (pass 2) of their scale, as for the stored chunks."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import golden_io as G
import tolerance as T
from oracle import kernels as OK
from test_kernels_gpu import EXACT, _block, _row_out

pytestmark = pytest.mark.gpu

SHAPES = [(3, 1), (4, 2), (5, 8), (9, 9), (10, 10), (13, 16), (15, 17), (16, 24), (17, 31), (17, 33), (23, 40), (31, 55),
          (33, 64), (41, 65)]


def _rows(case, bx, Dz, n, seed):
    """n boxes of bx x bx x Dz: a stored chunk's boxes pasted (or cropped) around the centre, on a Poisson background
    with masked, overloaded and unrecorded voxels and a few bright ones."""
    i = next(k for k in G.chunks(case) if G.chunk(case, k)[4])
    d, rc, nb, _, _ = G.chunk(case, i)
    m, Dz0, _, Dx0 = d["sb"].shape
    rng = np.random.default_rng(seed)
    pick = np.argsort(-rc["has_p"], kind="stable")[np.arange(n) % m] if case == "crowded" else np.arange(n) % m
    sb = rng.poisson(1.5, (n, Dz, bx, bx)).astype(np.float32)
    o, oz = bx // 2 - Dx0 // 2, Dz // 2 - Dz0 // 2
    dst = lambda off, size, full: (max(off, 0), min(off + size, full))
    (a, b), (c, e) = dst(o, Dx0, bx), dst(oz, Dz0, Dz)
    sb[:, c:e, a:b, a:b] = d["sb"][pick][:, c - oz:e - oz, a - o:b - o, a - o:b - o]
    flat = sb.reshape(n, -1)
    for r in range(n):
        if r % 3:
            flat[r, rng.choice(flat.shape[1], flat.shape[1] // 60, replace=False)] = -1.0
            flat[r, rng.choice(flat.shape[1], flat.shape[1] // 200, replace=False)] = -2.0
            flat[r, rng.choice(flat.shape[1], flat.shape[1] // 50, replace=False)] = 40.0
        if r % 4 == 3:
            sb[r, :max(Dz // 4, 1)] = -3.0
    one = {k: np.asarray(v)[pick].copy() for k, v in rc.items()}
    one["ix0"], one["iy0"], one["iz0"] = one["ix0"] - o, one["iy0"] - o, one["iz0"] - oz
    return d, sb, one, {k: np.asarray(v)[pick] for k, v in nb.items()}


@pytest.fixture
def tuned():
    from xpg_b200 import native as N
    lib = N.load()

    def tune(key, value):
        N.check(lib.xi_tune(key, value), "xi_tune")
    yield tune
    for key, value in ((N.XI_TUNE_WIDE_THREADS, 256), (N.XI_TUNE_PASS1_STAGE_BYTES, 48 * 1024),
                       (N.XI_TUNE_PASS2_STAGE_BYTES, 48 * 1024), (N.XI_TUNE_PASS2_LIST_CAP, 2048),
                       (N.XI_TUNE_PASS2_LIST_CAP_LARGE, 2048)):
        N.check(lib.xi_tune(key, value), "xi_tune")
    N._apply_tuned(lib)


@pytest.mark.parametrize("wide,stage,cap", [(256, 0, 2048), (256, 49152, 0), (128, 0, 24), (128, 49152, 2048)])
@pytest.mark.parametrize("case", ["config1", "crowded", "superpix"])
def test_shapes_match_oracle(case, wide, stage, cap, tuned):
    from xpg_b200 import device as D
    from xpg_b200 import native as N
    tuned(N.XI_TUNE_WIDE_THREADS, wide)
    tuned(N.XI_TUNE_PASS1_STAGE_BYTES, stage)
    tuned(N.XI_TUNE_PASS2_STAGE_BYTES, stage)
    tuned(N.XI_TUNE_PASS2_LIST_CAP, cap)
    tuned(N.XI_TUNE_PASS2_LIST_CAP_LARGE, cap)
    spec, tmpl, _, _ = G.case_inputs(case)
    det, odet = D.DeviceDetector(spec.geometry(), tmpl), OK.detector_consts(spec.geometry(), tmpl)
    n = 4
    for bx, Dz in SHAPES:
        d, sb, one, nb = _rows(case, bx, Dz, n, 100 * bx + Dz)
        pxs = one["pxs"].astype(np.int32) if "pxs" in one else np.ones(n, np.int32)
        rows = D.RowSet(**{k: one[k] for k in ("S", "phi", "ix0", "iy0", "iz0", "fb", "region", "has_p", "pS", "pphi")},
                        pxs=pxs, Dz=np.full(n, Dz), bx=np.full(n, bx), nb=nb, device="cuda", sb_bias=0.0)
        arena = torch.as_tensor(sb.reshape(-1)).cuda()
        blk, _k1 = _block(d)
        blk2, _k2 = _block(d, "p2_")
        p1, p2 = D.Pass1Buffers(rows), D.Pass2Buffers(rows)
        D.pass1(det, rows, blk, arena, p1)
        prof = torch.as_tensor(d["prof"]).cuda()
        D.pass2(det, rows, blk2, arena, prof, p1, p2)
        D.status()
        h1, h2 = ({k: v.cpu().numpy() for k, v in q.t.items()} for q in (p1, p2))
        for j in range(n):
            mine, r, q = _row_out(h1, rows, j), G.row_dict(one, j), G.nb_row(nb, j)
            ref = OK.pass1(sb[j], r, q, odet, d["s0"], d["axis"], d["frames_phi0"], d["osc"], d["sd"], d["sm"], d["gain"],
                           d["rcw"])
            for k in EXACT:
                assert np.array_equal(np.asarray(mine[k], np.float64), np.asarray(ref[k], np.float64)), (bx, Dz, j, k)
            for k in ("isum", "vsum", "vsum0", "xo", "yo", "zo", "m_d", "m_m", "frac_rec", "img2", "fz"):
                ok, worst = T.within(k, mine[k], ref[k], ref, rel=1e-5)
                assert ok, (bx, Dz, j, k, worst)
            pix = {k: mine[k] for k in ("zeta", "J", "u1", "u2", "seff")}
            want = OK.pass2(sb[j], r, q, odet, d["s0"], d["axis"], d["frames_phi0"], d["osc"], d["p2_sd"], d["p2_sm"],
                            d["p2_gain"], d["prof"], mine["bg"], mine["nbg"], d["p2_rcw"], pix)
            for k in want:
                ok, worst = T.within(k, h2[k][j], want[k], dict(want, vsum=mine["vsum"]), rel=2e-6)
                assert ok, (bx, Dz, j, k, worst, h2[k][j], want[k])
