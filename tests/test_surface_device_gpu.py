"""make_kernels on arguments that are already device tensors (any dtype or stride) gives the bits it gives on the same
values as numpy arrays."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import golden_io as G

pytestmark = pytest.mark.gpu


def _wide(a):
    """A strided device view of wider elements that hold the same values."""
    a = np.asarray(a)
    t = torch.as_tensor(a).cuda()
    t = t.double() if t.is_floating_point() else t.long()
    return torch.stack([t, torch.zeros_like(t)], -1)[..., 0]


@pytest.mark.parametrize("put", [lambda a: torch.as_tensor(np.asarray(a)).cuda(), _wide], ids=["plain", "strided"])
def test_device_arguments_match_host_arguments(put):
    from xpg_b200.kernels import detector_consts, make_kernels
    case = "crowded"
    spec, tmpl, _, _ = G.case_inputs(case)
    d, rc, nb, _, _ = G.chunk(case, 0)
    Dz, Dy, Dx = (int(v) for v in d["shape"])
    p1, acc, p2 = make_kernels(Dz, Dy, Dx, spec.n_regions_xy ** 2)
    det = detector_consts(spec.geometry(), tmpl)
    sel = np.arange(d["sb"].shape[0]) % 2 == 0

    def run(f):
        sb, r, q = f(d["sb"]), {k: f(v) for k, v in rc.items()}, {k: f(v) for k, v in nb.items()}
        o = p1(sb, r, det, d["axis"], d["s0"], d["frames_phi0"], d["osc"], d["sd"], d["sm"], d["gain"], None, q,
               f(d["rcw"]))
        get = (lambda k: o[k].cpu().numpy()) if f is np.asarray else (lambda k: f(o[k].cpu().numpy()))
        num, den = acc(*(get(k) for k in ("img2", "all_valid2", "J", "u1", "u2")), r["region"], get("isum"), f(sel),
                       get("seff"))
        fit = p2(sb, r, det, d["axis"], d["s0"], d["frames_phi0"], d["osc"], d["p2_sd"], d["p2_sm"], d["p2_gain"],
                 f(d["prof"]), get("bg"), get("nbg"), q, f(d["p2_rcw"]),
                 {k: get(k) for k in ("zeta", "J", "u1", "u2", "seff")})
        return {k: v for k, v in o.items() if not k.startswith("_")}, (num, den), fit
    host, dev = run(np.asarray), run(put)
    for a, b in ((host[0], dev[0]), (host[2], dev[2])):
        for k in a:
            assert torch.equal(a[k].double().nan_to_num(7.0), b[k].double().nan_to_num(7.0)), k
    for a, b in zip(host[1], dev[1]):                      # float64 sums added in any order: a few last bits
        torch.testing.assert_close(a, b, rtol=1e-12, atol=1e-12)
