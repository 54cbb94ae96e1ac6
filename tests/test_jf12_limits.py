"""Breg_jf12 at its limits.  Over the X-field angles that the model takes: level
(the radius that bounds the inner region is infinite off the plane), steep, and
beyond a right angle or below zero, where the inner region's angle changes sign.
Faraday depth maps of an exponential disk against a plain numpy sum of the
reference's expressions (breg_jf12.cc:72-186): 1e-10 of the map maximum in FP64
(the parity suite's bar), 1e-5 in FP32C."""
import math

import numpy as np
import pytest

from conftest import rel_err
from hammurabix_b200 import abi, units as U, workloads as W

JF12 = dict(b_arm1=0.1, b_arm2=3.0, b_arm3=-0.9, b_arm4=-0.8, b_arm5=-2.0, b_arm6=-4.2,
            b_arm7=0.0, b_ring=0.1, h_disk=0.40, w_disk=0.27, Bn=1.4, Bs=-1.1, rn=9.22,
            rs=16.7, wh=0.2, z0=5.3, B0_X=4.6, rpc_X=4.8, r0_X=2.9)
LENGTHS = ("h_disk", "w_disk", "rn", "rs", "wh", "z0", "rpc_X", "r0_X")
ANGLES = [0.0, 20.0, 120.0, 165.0, -30.0]


def _models(angle):
    m = W.spiral_models()
    m.breg = abi.HXG_BREG_JF12
    for k, v in JF12.items():
        setattr(m.jf12, k, v * (U.kpc if k in LENGTHS else U.muGauss))
    m.jf12.Xtheta = angle * U.rad
    return m


def _field(x, y, z, angle):
    """Cartesian B in muG at positions in kpc (breg_jf12.cc:35-190)."""
    p = JF12
    r, phi, az = np.hypot(x, y), np.arctan2(y, x), np.abs(z)
    zp = 1 / (1 + np.exp(-2 / p["w_disk"] * (az - p["h_disk"])))
    f = [0.130, 0.165, 0.094, 0.122, 0.13, 0.118, 0.084, 0.156]
    rc = [5.1, 6.3, 7.1, 8.3, 9.8, 11.4, 12.7, 15.5]
    bv = [p[f"b_arm{k}"] for k in range(1, 8)]
    bv.append(-sum(a * b for a, b in zip(f, bv)) / f[7])
    inc = math.radians(11.5)
    cot = 1 / math.tan(math.radians(90 - 11.5))
    rn = r * np.exp(-cot * (phi - np.pi))
    rn = np.where(rn > rc[7], r * np.exp(-cot * (phi + np.pi)), rn)
    rn = np.where(rn > rc[7], r * np.exp(-cot * (phi + 3 * np.pi)), rn)
    arm = np.zeros_like(r)
    for k in range(7, -1, -1):
        arm = np.where(rn < rc[k], bv[k], arm)
    b0 = 5 / r * (1 - zp)
    br = np.where(r >= 5, arm * b0 * math.sin(inc), 0)
    bp = np.where(r >= 5, arm * b0 * math.cos(inc), np.where(r > 3, b0 * p["b_ring"], 0))
    b1, rh = np.where(z >= 0, p["Bn"], p["Bs"]), np.where(z >= 0, p["rn"], p["rs"])
    bp = bp + zp * b1 * (1 - 1 / (1 + np.exp(-2 / p["wh"] * (r - rh)))) * np.exp(-az / p["z0"])
    tx = np.float64(math.tan(math.radians(angle)))
    with np.errstate(all="ignore"):
        rcx = p["rpc_X"] + az / tx
        inner = r < rcx
        rp = np.where(inner, r * p["rpc_X"] / rcx, r - az / tx)
        bx = p["B0_X"] * np.where(inner, (p["rpc_X"] / rcx) ** 2, rp / r) * np.exp(-rp / p["r0_X"])
        ang = np.where(inner, np.arctan(az / (r - rp)), math.radians(angle))
    br = br + bx * np.cos(ang) * np.where(z < 0, -1, 1)
    out = (r > 20) | (np.sqrt(r * r + z * z) < 1)
    c, s = x / r, y / r
    return [np.where(out, 1e-6, v) for v in (br * c - bp * s, br * s + bp * c, bx * np.sin(ang))]


def _fd(oracle, o, angle):
    """Faraday depth map of the one shell of o.  Positions in extended precision and
    rounded once, as a fused multiply-add gives them: samples can lie on a cut."""
    th, ph = oracle.pix2ang(o.nside_shell[0])
    d_start, delta, n = oracle.shell_ref(o, 0)
    u = [np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)]
    fma = lambda a, b, c: (a.astype(np.longdouble) * b + c).astype(np.float64)  # noqa: E731
    d = fma(np.arange(n) + 0.5, delta, d_start)
    pos = [fma(a[:, None], d, o.observer[k]) for k, a in enumerate(u)]
    on = (np.sqrt(sum(c * c for c in pos)) <= o.gc_r_max) & (np.abs(pos[2]) <= o.gc_z_max)
    x, y, z = (c / U.kpc for c in pos)
    ne = 0.03 * np.exp(-np.hypot(x, y) / 20 - np.abs(z))
    bpar = sum(b * a[:, None] for b, a in zip(_field(x, y, z, angle), u)) * 1e-6
    qe, mec2 = 4.80320425e-10, 0.51099907e-3 * 1.60217733e-12 * 1e9
    return -qe ** 3 / (2 * math.pi * mec2 ** 2) * delta * np.where(on, ne * bpar, 0).sum(1)


@pytest.mark.gpu
@pytest.mark.parametrize("angle", ANGLES)
@pytest.mark.parametrize("form,tol", [("fp64", 1e-10), ("fp32c", 1e-5)])
def test_faraday_depth_vs_numpy(oracle, form, tol, angle):
    from hammurabix_b200.integrator import Integrator
    for observer in (W.OBSERVER_KPC, (0.5, -0.3, 9.0)):
        o = W.make_obs([8], 24.0, 0.1, observer_kpc=observer, do_dm=False)
        with Integrator(form) as ig:
            ig.set_models(_models(angle))
            got = ig.write_grid(o)["fd"]
        assert np.isfinite(got).all()
        assert rel_err(got, _fd(oracle, o, angle)) <= tol, observer


@pytest.mark.gpu
@pytest.mark.parametrize("alpha", [1.0, 2.7, 3.0])
def test_beyond_the_halo_edge(alpha):
    """Without an X field nothing is left some wh beyond the halo's edge: the sky
    there is empty and finite, and both forms agree (1e-5, the FP32C bar)."""
    from hammurabix_b200.integrator import Integrator
    m = _models(49.0)
    m.jf12.B0_X = 0.0
    m.cre_ana.alpha = alpha
    o = W.make_obs([8], 24.0, 0.05, freq_ghz=23.0, observer_kpc=(-16.0, 0.0, 3.0))
    got = {}
    for form in ("fp64", "fp32c"):
        with Integrator(form) as ig:
            ig.set_models(m)
            got[form] = ig.write_grid(o)
    for k, a in got["fp64"].items():
        assert np.isfinite(a).all() and np.abs(a).max() > 0 and a.min() > -1e20, k
        assert rel_err(got["fp32c"][k], a) <= 1e-5, k
