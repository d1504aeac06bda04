"""XPG's inner kernel surface on the B200 kernels: `make_kernels(Dz, Dy, Dx, n_regions, G=41)` returns
(pass1, accumulate_profiles, pass2) with the reference's signatures and dict results
(`xpg/integrate_kernels.py:216-485`), for callers that drive the kernels themselves.

Arguments are torch CUDA tensors, read where they are (anything else is moved to the device): `sb` (N, Dz, Dy, Dx) float32 shoeboxes
(values, -1 masked, -2 overloaded, -3 unrecorded), the `rc` dict (S, phi, ix0, iy0, iz0, fb, region, has_p, pS, pphi
and optionally pxs), the `nb` dict (x, y, z, sx, sz: (N, K)), and `det` from `detector_consts(geometry,
bkg_template)` (XPG's `_detector_consts`). `axis`, `s0`, `frames_phi0`, `osc`, `sd`, `sm`, `gain` and `rcw` as in the
reference. Only Dy == Dx boxes exist in XPG and here.
"""
from __future__ import annotations

import numpy as np
import torch

from . import device as D
from . import native as N

PROFILE_GRID = 41


def detector_consts(g, bkg_template=None, device="cuda"):
    """Device detector description of a geometry (`xpg/integrate_kernels.py:48-65`)."""
    return D.DeviceDetector(g, bkg_template, device)


def _np(v):
    if torch.is_tensor(v):
        return v.detach().cpu().numpy()
    return np.asarray(v)


# the types of tensors that have a numpy form (bfloat16, float8 and views with a pending conjugate or sign have none)
_TYPES = frozenset((torch.float64, torch.float32, torch.float16, torch.int64, torch.int32, torch.int16, torch.int8,
                    torch.uint64, torch.uint32, torch.uint16, torch.uint8, torch.bool, torch.complex64,
                    torch.complex128))


def _in(v):
    """A per-row or per-pixel argument for `device._dev`: a CUDA tensor as it is (it is converted on the device, or
    read in place), anything else as a numpy array. Through the host instead, the pixel tables' copies alone took
    most of a call (4096 boxes of 31 x 31 x 33: 26.3 ms for the three passes, 3.8 ms of it kernels)."""
    if not (torch.is_tensor(v) and v.is_cuda):
        return _np(v)
    if v.dtype not in _TYPES or v.is_neg() or (v.dtype.is_complex and v.is_conj()):
        raise TypeError(f"a {v.dtype} tensor without a numpy form (its type, or a pending sign or conjugate)")
    return v.detach() if v.requires_grad else v


def _as(v, dtype):
    """`_in`, a numpy array converted to `dtype` by numpy (which takes foreign byte orders and long doubles)."""
    v = _in(v)
    return v if torch.is_tensor(v) else v.astype(dtype)


def _on_device(v):
    """The argument's values as a device tensor, in its own shape."""
    t = _in(v)
    return t.to("cuda") if torch.is_tensor(t) else torch.as_tensor(t).to("cuda")


def _rows(sb, rc, nb, Dz, Dx):
    n = int(sb.shape[0])
    one = ("S", "phi", "ix0", "iy0", "iz0", "fb", "region", "has_p", "pS", "pphi")
    pxs = _as(rc["pxs"], np.int32) if "pxs" in rc else np.ones(n, np.int32)
    return D.RowSet(**{k: _in(rc[k]) for k in one}, pxs=pxs, Dz=np.full(n, Dz), bx=np.full(n, Dx),
                    nb={k: _in(nb[k]) for k in ("x", "y", "z", "sx", "sz")}, sb_bias=0.0)


def _block(axis, s0, frames_phi0, osc, sd, sm, gain, rcw):
    b = N.XiBlock()
    b.frames_phi0, b.osc = float(np.float32(frames_phi0)), float(np.float32(osc))
    b.sd, b.sm, b.gain = float(np.float32(sd)), float(np.float32(sm)), float(np.float32(gain))
    rc = torch.as_tensor(_np(rcw).astype(np.float32)).cuda()
    b.rcw = N.ptr(rc)
    a, s = _np(axis).astype(np.float32), _np(s0).astype(np.float32)
    for c in range(3):
        b.axis[c], b.s0[c] = float(a[c]), float(s[c])
    return b, rc


def _groups(rows):
    """One launch over the rows in order: they have one shape."""
    return [(int(rows.bx[0]), int(rows.Dz[0]), None)] if rows.n else []


def _sb(sb):
    t = torch.as_tensor(sb) if not torch.is_tensor(sb) else sb
    return t.to("cuda", torch.float32).contiguous().reshape(-1)


def make_kernels(Dz, Dy, Dx, n_regions, G=PROFILE_GRID):
    if Dy != Dx:
        raise ValueError("square boxes only (Dy == Dx)")
    if G != PROFILE_GRID:
        raise ValueError("the kernels use the 41 x 41 profile grid")
    N.require_cuda()

    def pass1(sb, rc, det, axis, s0, frames_phi0, osc, sd, sm, gain, prof, nb, rcw):
        """Background, summation, centroids, 2D projected spot images (`xpg/integrate_kernels.py:287-365`)."""
        rows = _rows(sb, rc, nb, Dz, Dx)
        blk, keep = _block(axis, s0, frames_phi0, osc, sd, sm, gain, rcw)
        arena = _sb(sb)
        out = D.Pass1Buffers(rows)
        D.pass1(det, rows, blk, arena, out, groups=_groups(rows))
        D.status()
        t = out.t
        n = rows.n
        res = {k: t[k] for k in D.Pass1Buffers.SCALARS if k not in ("zeta", "seff")}
        res.update({k: t[k] for k in D.Pass1Buffers.COUNTS})
        res["fz"] = t["fz"].view(n, Dz)
        res["img2"] = t["img2"].view(n, Dy, Dx)
        res["all_valid2"] = t["all_valid2"].view(n, Dy, Dx).bool()
        res["zeta"], res["seff"] = t["zeta"], t["seff"]
        res["J"] = t["J"].view(n, Dy, Dx)
        res["u1"] = t["u1"].view(n, Dy, Dx)
        res["u2"] = t["u2"].view(n, Dy, Dx)
        res["_rows"] = rows
        res["_buf"] = out
        return res

    def accumulate_profiles(img2, ok2, J, u1, u2, region, isum, sel, seff):
        """Normalised projected spots scattered into per-region float64 grids (`:367-380`)."""
        n = int(img2.shape[0])
        nbz = {k: np.zeros((n, 1), np.float32) for k in ("x", "y", "z", "sx", "sz")}
        rc = dict(S=np.zeros((n, 3), np.float32), phi=np.zeros(n, np.float32), ix0=np.zeros(n, np.int32),
                  iy0=np.zeros(n, np.int32), iz0=np.zeros(n, np.int32), fb=np.ones(n, np.float32), region=_in(region),
                  has_p=np.zeros(n, np.float32), pS=np.zeros((n, 3), np.float32), pphi=np.zeros(n, np.float32))
        rows = _rows(np.zeros((n, 1, Dy, Dx), np.float32), rc, nbz, 1, Dx)
        buf = D.Pass1Buffers(rows)
        for k, v in (("img2", img2), ("J", J), ("u1", u1), ("u2", u2)):
            buf.t[k].copy_(_on_device(v).reshape(-1).float())
        buf.t["all_valid2"].copy_(_on_device(ok2).reshape(-1).to(torch.uint8))
        buf.t["isum"].copy_(_on_device(isum).float())
        buf.t["seff"].copy_(_on_device(seff).float())
        num = torch.zeros((n_regions, G, G), dtype=torch.float64, device="cuda")
        den = torch.zeros_like(num)
        selt = _on_device(sel).to(torch.uint8).contiguous()
        D.accumulate(rows, buf, n_regions, num, den, sel=selt, strong_test=False)
        for v in (img2, ok2, J, u1, u2, region, isum, sel, seff):      # read behind the call's return
            if torch.is_tensor(v) and v.is_cuda:
                v.record_stream(torch.cuda.current_stream(v.device))
        return num, den

    def pass2(sb, rc, det, axis, s0, frames_phi0, osc, sd, sm, gain, prof, bg, nbm_x, nb, rcw, pix=None):
        """Profile fit with fixed background and the joint fit of overlapping partners (`:382-483`). `pix`: pass 1's
        zeta / J / u1 / u2 / seff of these rows (computed here when absent)."""
        rows = _rows(sb, rc, nb, Dz, Dx)
        arena = _sb(sb)
        if pix is None:
            r1 = pass1(sb, rc, det, axis, s0, frames_phi0, osc, sd, sm, gain, prof, nb, rcw)
            pix = {k: r1[k] for k in ("zeta", "J", "u1", "u2", "seff")}
        buf = D.Pass1Buffers(rows)
        for k, v in (*((k, pix[k]) for k in ("zeta", "seff", "J", "u1", "u2")), ("bg", bg), ("nbg", nbm_x)):
            buf.t[k].copy_(_on_device(v).reshape(-1).float())
        blk, keep = _block(axis, s0, frames_phi0, osc, sd, sm, gain, rcw)
        out = D.Pass2Buffers(rows)
        proft = _on_device(_as(prof, np.float32)).float().contiguous()
        D.pass2(det, rows, blk, arena, proft, buf, out, groups=_groups(rows))
        D.status()
        return dict(out.t)

    return pass1, accumulate_profiles, pass2
