"""The forward passes at both work splits (a warp or a CTA a reflection, on either side of the count where the rule
changes), one to four terms, odd sides, boxes across every border of the window and wholly outside it, counts of every
type with zeros and masked voxels, against the oracle: float32 sums in another order, within 1e-5 of scale."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import forward as OF
from test_forward import RTOL

pytestmark = pytest.mark.gpu


class _Win:
    def __init__(self, w):
        self.f0, self.f1, self.y0, self.ny, self.x0, self.nx = (int(v) for v in w)


@pytest.mark.parametrize("n,terms,Dz,b,counts", [(1, 1, 1, 1, "int16"), (33, 3, 5, 4, "int32"), (9471, 2, 3, 5, "int16"),
                                                 (9472, 2, 5, 5, "int16"), (9475, 1, 4, 7, "float32"),
                                                 (9500, 4, 6, 3, "int32"), (40, 2, 9, 21, "float32")])
def test_passes_match_oracle(n, terms, Dz, b, counts):
    from xpg_b200 import forward as F
    rng = np.random.default_rng(n + 10 * terms)
    w = (4, 17, 30, 40, 50, 45)                            # f0, f1, y0, ny, x0, nx
    nv = (w[1] - w[0]) * w[3] * w[5]
    R = rng.uniform(0.0, 0.5, (terms, n, Dz)).astype(np.float32)
    P = rng.uniform(0.0, 0.1, (terms, n, b, b)).astype(np.float32)
    iz0 = rng.integers(w[0] - Dz - 1, w[1] + 2, n)
    iy0 = rng.integers(w[2] - b - 1, w[2] + w[3] + 2, n)
    ix0 = rng.integers(w[4] - b - 1, w[4] + w[5] + 2, n)
    I, beta = rng.uniform(0, 50, n).astype(np.float32), rng.uniform(0, 0.1, n).astype(np.float32)
    B0 = rng.uniform(0.1, 0.4, nv).astype(np.float32)
    NS = rng.poisson(0.5, nv).astype(np.float32)
    NS[rng.random(nv) < 0.05] = -1.0
    A, M = np.maximum(NS, 0.0), rng.uniform(0.2, 3.0, nv).astype(np.float32)
    rows = rng.permutation(n)
    grp = [dict(R=R, P=P, iz0=iz0, iy0=iy0, ix0=ix0, rows=rows)]
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()
    box, at = (t(R), t(P)), (t(iz0), t(iy0), t(ix0), _Win(w))
    mu = t(B0)
    F.scatter(mu, *box, t(I[rows]), t(beta[rows]), *at)
    g = torch.zeros((3, n), device="cuda")
    ns = t(NS).to(getattr(torch, counts))
    F.gather(g[0], None, *box, t(rows), *at, t(A), t(M), ns, 0)
    F.gather(g[1], g[2], *box, t(rows), *at, None, t(M), ns, 1)
    ratio, _ = OF.gather(grp, w, n, A, M, NS, 0)
    newton, fisher = OF.gather(grp, w, n, None, M, NS, 1)
    for got, want, floor in ((mu, OF.scatter(B0, grp, I, beta, w), 1.0), (g[0], ratio, 1e-3), (g[1], newton, 1e-3),
                             (g[2], fisher, 1e-3)):
        scale = np.maximum(np.abs(want), floor)
        assert (np.abs(got.cpu().numpy().reshape(want.shape) - want) <= RTOL * scale).all()
