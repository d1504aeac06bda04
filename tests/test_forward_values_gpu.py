"""The forward gathers on models that are zero, negative, infinite or NaN (the quotients' special cases: zero counts take
a path of their own), and the work split of small boxes on either side of its counts, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import test_forward_rows_gpu as rows
from oracle import forward as OF
from test_forward import RTOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,terms,Dz,b,counts", [(300, 2, 4, 5, "int16"), (1183, 1, 3, 8, "int32"),
                                                 (1184, 2, 3, 8, "float32"), (1200, 3, 5, 6, "int16"),
                                                 (1184, 1, 4, 9, "int16")])
def test_small_boxes_match_oracle(n, terms, Dz, b, counts):
    rows.test_passes_match_oracle(n, terms, Dz, b, counts)


@pytest.mark.parametrize("n,b", [(40, 9), (3000, 5), (9500, 7)])
@pytest.mark.parametrize("value", [0.0, -0.5, np.inf, np.nan])
def test_special_models_match_oracle(value, n, b):
    from xpg_b200 import forward as F
    rng = np.random.default_rng(n + b)
    w = (4, 17, 30, 40, 50, 45)                            # f0, f1, y0, ny, x0, nx
    Dz, nv = 5, 13 * 40 * 45
    R = rng.uniform(0.1, 0.5, (2, n, Dz)).astype(np.float32)
    P = rng.uniform(0.01, 0.1, (2, n, b, b)).astype(np.float32)
    at = [rng.integers(lo - 2, lo + size + 2, n) for lo, size in ((4, 13), (30, 40), (50, 45))]
    NS = rng.poisson(0.5, nv).astype(np.float32)
    NS[rng.random(nv) < 0.05] = -1.0
    A, M = np.maximum(NS, 0.0), rng.uniform(0.2, 3.0, nv).astype(np.float32)
    M[rng.choice(nv, 60, replace=False)] = np.float32(value)
    grp = [dict(R=R, P=P, iz0=at[0], iy0=at[1], ix0=at[2], rows=np.arange(n))]
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()
    box, place = (t(R), t(P)), (*(t(a) for a in at), rows._Win(w))
    g = torch.zeros((3, n), device="cuda")
    ns = t(NS).to(torch.int16)
    F.gather(g[0], None, *box, t(np.arange(n)), *place, t(A), t(M), ns, 0)
    F.gather(g[1], g[2], *box, t(np.arange(n)), *place, None, t(M), ns, 1)
    with np.errstate(all="ignore"):
        ratio, _ = OF.gather(grp, w, n, A, M, NS, 0)
        newton, fisher = OF.gather(grp, w, n, None, M, NS, 1)
        ratio, newton = ratio.astype(np.float32), newton.astype(np.float32)
    pairs = [(g[0], ratio), (g[1], newton)]
    if not np.isnan(value):                                # (the kernel's floor of the model takes a NaN away)
        pairs.append((g[2], fisher))
    for got, want in pairs:
        got, want = got.cpu().numpy().astype(np.float64), want.astype(np.float64)
        odd = ~np.isfinite(want)
        assert np.array_equal(got[odd], want[odd], equal_nan=True)
        assert (np.abs(got[~odd] - want[~odd]) <= RTOL * np.maximum(np.abs(want[~odd]), 1e-3)).all()
