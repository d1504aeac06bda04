"""make_kernels' argument types: what numpy converts (foreign byte order, long double) is taken, and device tensors that
have no numpy form (bfloat16, views with a pending sign) are refused, as when every argument went through numpy."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import golden_io as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def call():
    from xpg_b200.kernels import detector_consts, make_kernels
    spec, tmpl, _, _ = G.case_inputs("crowded")
    d, rc, nb, _, _ = G.chunk("crowded", 0)
    Dz, Dy, Dx = (int(v) for v in d["shape"])
    p1, _, p2 = make_kernels(Dz, Dy, Dx, spec.n_regions_xy ** 2)
    det = detector_consts(spec.geometry(), tmpl)

    def run(prof=d["prof"], n=None, **one):
        sb, r, q = d["sb"][:n], {k: v[:n] for k, v in {**rc, **one}.items()}, {k: v[:n] for k, v in nb.items()}
        o = p1(sb, r, det, d["axis"], d["s0"], d["frames_phi0"], d["osc"], d["sd"], d["sm"], d["gain"], None, q, d["rcw"])
        return p2(sb, r, det, d["axis"], d["s0"], d["frames_phi0"], d["osc"], d["p2_sd"], d["p2_sm"], d["p2_gain"], prof,
                  o["bg"], o["nbg"], q, d["p2_rcw"], {k: o[k] for k in ("zeta", "J", "u1", "u2", "seff")})
    return run, d, rc


@pytest.mark.parametrize("kind", [">f4", ">f8", np.longdouble])
def test_profiles_that_numpy_converts(call, kind):
    run, d, _ = call
    want, got = run(), run(prof=np.asarray(d["prof"]).astype(kind))
    assert torch.equal(got["iprf"], want["iprf"])


@pytest.mark.parametrize("kind", [">i4", ">i8", np.longdouble])
def test_superpixel_sides_that_numpy_converts(call, kind):
    run, d, _ = call
    pxs = np.ones(len(d["sb"]))
    assert torch.equal(run(pxs=pxs.astype(kind))["iprf"], run(pxs=pxs.astype(np.int32))["iprf"])


def test_device_tensors_without_a_numpy_form_are_refused(call):
    run, d, rc = call
    with pytest.raises(TypeError):
        run(prof=torch.as_tensor(d["prof"]).cuda().bfloat16())
    with pytest.raises(TypeError):
        run(phi=torch.as_tensor(rc["phi"]).cuda().bfloat16())
    z = torch.complex(torch.zeros(len(rc["phi"])), -torch.as_tensor(rc["phi"])).cuda().conj().imag
    assert z.is_neg()
    with pytest.raises(TypeError):
        run(n=1, phi=z)
