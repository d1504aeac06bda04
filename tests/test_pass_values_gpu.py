"""Pass 1 and pass 2 where a box's values or its spot take them off their common path: backgrounds that all lie above the
lowest clip threshold (the list of clip candidates overflows), scattered masked voxels, NaN voxels (not valid, not
recorded), and spots so wide that the fitted voxels overflow their list, with the candidate pixels inside or beyond
theirs. Against the oracle: masks, counts, background and per-pixel terms bit for bit, sums within 1e-5 of their scale."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import golden_io as G
import tolerance as T
from oracle import kernels as OK
from test_kernels_gpu import EXACT, _block, _row_out
from test_pass_shapes_gpu import _rows, tuned  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

SUMS = ("isum", "vsum", "vsum0", "xo", "yo", "zo", "frac_rec", "img2", "fz")


def _run(case, d, sb, one, nb, widen=1.0, sm=None):
    """Both passes of the boxes on the device and by the oracle (spot widths times `widen`, rocking width `sm`)."""
    from xpg_b200 import device as D
    spec, tmpl, _, _ = G.case_inputs(case)
    det, odet = D.DeviceDetector(spec.geometry(), tmpl), OK.detector_consts(spec.geometry(), tmpl)
    n, Dz, bx, _ = sb.shape
    pxs = one["pxs"].astype(np.int32) if "pxs" in one else np.ones(n, np.int32)
    rows = D.RowSet(**{k: one[k] for k in ("S", "phi", "ix0", "iy0", "iz0", "fb", "region", "has_p", "pS", "pphi")},
                    pxs=pxs, Dz=np.full(n, Dz), bx=np.full(n, bx), nb=nb, device="cuda", sb_bias=0.0)
    arena = torch.as_tensor(sb.reshape(-1)).cuda()
    sd = np.float32(d["sd"] * widen)
    sm = np.float32(d["sm"] if sm is None else sm)
    blk, _keep = _block(d)
    blk.sd, blk.sm = float(sd), float(sm)
    p1, p2 = D.Pass1Buffers(rows), D.Pass2Buffers(rows)
    D.pass1(det, rows, blk, arena, p1)
    D.pass2(det, rows, blk, arena, torch.as_tensor(d["prof"]).cuda(), p1, p2)
    D.status()
    h1, h2 = ({k: v.cpu().numpy() for k, v in q.t.items()} for q in (p1, p2))
    for j in range(n):
        mine, r, q = _row_out(h1, rows, j), G.row_dict(one, j), G.nb_row(nb, j)
        at = (odet, d["s0"], d["axis"], d["frames_phi0"], d["osc"], sd, sm, d["gain"])
        ref = OK.pass1(sb[j], r, q, *at, d["rcw"])
        pix = {k: mine[k] for k in ("zeta", "J", "u1", "u2", "seff")}
        want = OK.pass2(sb[j], r, q, *at, d["prof"], mine["bg"], mine["nbg"], d["rcw"], pix)
        yield j, mine, ref, {k: h2[k][j] for k in want}, want


def _compare(name, rows):
    for j, mine, ref, fit, want in rows:
        for k in EXACT:
            assert np.array_equal(np.asarray(mine[k], np.float64), np.asarray(ref[k], np.float64)), (name, j, k)
        for k in SUMS:
            ok, worst = T.within(k, mine[k], ref[k], ref, rel=1e-5)
            assert ok, (name, j, k, worst)
        for k in want:
            ok, worst = T.within(k, fit[k], want[k], dict(want, vsum=mine["vsum"]), rel=1e-5)
            assert ok, (name, j, k, worst, fit[k], want[k])


@pytest.mark.parametrize("stage", [0, 49152])
@pytest.mark.parametrize("bx,Dz", [(9, 9), (17, 33), (23, 17), (31, 10), (41, 65)])
@pytest.mark.parametrize("case", ["config1", "crowded", "superpix"])
def test_bright_masked_and_nan_boxes(case, bx, Dz, stage, tuned):
    from xpg_b200 import native as N
    tuned(N.XI_TUNE_PASS1_STAGE_BYTES, stage)
    tuned(N.XI_TUNE_PASS2_STAGE_BYTES, stage)
    d, sb, one, nb = _rows(case, bx, Dz, 4, 7 * bx + Dz)
    rng = np.random.default_rng(bx + Dz)
    level = np.array([25.0, 3.0, 25.0, 0.0])[:, None, None, None]      # all above the threshold, some, all, few
    sb = np.where(sb >= 0, sb + rng.poisson(level, sb.shape), sb).astype(np.float32)
    sb[2][rng.random(sb.shape[1:]) < 0.3] = -1.0
    sb[3][rng.random(sb.shape[1:]) < 0.03] = np.nan
    _compare((case, bx, Dz), _run(case, d, sb, one, nb))


@pytest.mark.parametrize("wide,cap", [(256, 2048), (256, 0), (128, 2048)])
@pytest.mark.parametrize("bx,Dz,pixels,voxels", [(31, 33, 0, 7000), (41, 65, 0, 20000), (73, 17, 2048, 20000),
                                                 (97, 1, 2048, 4000), (97, 65, 2048, 50000)])
def test_wide_spots(bx, Dz, pixels, voxels, wide, cap, tuned):
    """Spots that fill their boxes: more fitted voxels than any list of the shape holds, and of 97 px boxes more
    candidate pixels than the pixel list."""
    from xpg_b200 import native as N
    tuned(N.XI_TUNE_WIDE_THREADS, wide)
    tuned(N.XI_TUNE_PASS2_LIST_CAP, cap)
    tuned(N.XI_TUNE_PASS2_LIST_CAP_LARGE, cap)
    d, sb, one, nb = _rows("crowded", bx, Dz, 3, bx + Dz)
    one["has_p"] = np.array([1.0, 0.0, 1.0], np.float32) * (one["has_p"] > 0.5)
    nb = {k: v.copy() for k, v in nb.items()}
    for k in ("sx", "sz"):
        nb[k][:2] *= np.float32(0.01)                      # (neighbours of the third row only)
    spec, tmpl, _, _ = G.case_inputs("crowded")
    odet = OK.detector_consts(spec.geometry(), tmpl)
    r = G.row_dict(one, 0)
    gt = OK.geometry(odet, r, (Dz, bx, bx), d["s0"], d["axis"], d["frames_phi0"], d["osc"], d["sd"], d["sm"], d["rcw"])
    widen = abs(float(gt["u1"][bx // 2, 0])) / 2.2
    sm = abs(float(gt["zeta"])) * float(d["osc"]) * max(Dz, 3) / 6.0
    gt = OK.geometry(odet, r, (Dz, bx, bx), d["s0"], d["axis"], d["frames_phi0"], d["osc"], d["sd"] * widen, sm, d["rcw"])
    plane = OK.profile_plane(d["prof"][int(r["region"])], gt)
    p = plane[None] * gt["R"][:, None, None]
    assert (p > 0.01 * p.max()).sum() > voxels and (p.max(0) > 0.01 * p.max()).sum() > pixels
    _compare((bx, Dz, wide, cap), _run("crowded", d, sb, one, nb, widen, sm))
