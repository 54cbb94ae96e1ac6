"""Timed cases of the line-of-sight integrator: what its users run, through the
public Python entry points (hammurabix_b200.integrator, .autograd).

A case is a dict of plain values.  Common keys:

  kind    what the call is:
            "host"      Integrator.write_grid_multi into new numpy maps
            "upload"    FP32 host grids uploaded, then maps into pinned memory
            "device"    Integrator.write_grid_multi_device into torch tensors
            "adjoint"   autograd.LOSMaps forward, a least-squares loss, backward
            "batch"     Integrator.batch(...).run() over many parameter sets
            "generate"  random B and n_e fields generated, then one pass
  form    "fp64" (parity form, the default of the API) or "fp32c"
  fields  "spiral" (analytic), "grid" (spiral + B_rnd grid, n_e grid),
          "jf12" (JF12 regular field + B_rnd grid, n_e grid)
  nsides  Nside of the shells, innermost first; outputs at the largest
  r_max, res (kpc); freqs (GHz, the order of the <sync> list); grid "NXxNYxNZ"
  alpha   CRE spectral index; mask: Nside of the sky mask, 0 for none

Sizes are those of this repository's workloads (hammurabix_b200/workloads.py,
bench.py) and test cases, or generic.
"""
import math

import numpy as np
import torch

from hammurabix_b200 import abi, workloads
from hammurabix_b200 import units as U
from hammurabix_b200.autograd import LOSMaps
from hammurabix_b200.integrator import Integrator

KEYS = ("dm", "fd", "is", "qs", "us")
# 1-sigma scales of the least-squares loss: cm^-2, rad cm^-2, K (23 GHz)
LOSS_SCALE = (3e20, 1e-2, 1e-3, 3e-4, 3e-4)


def _case(name, kind, form, fields, nsides, r_max, res, freqs, grid="", alpha=3.0, mask=0,
          sets=0):
    c = dict(kind=kind, form=form, fields=fields, nsides=",".join(map(str, nsides)),
             r_max=float(r_max), res=float(res), freqs=",".join(map(str, freqs)), grid=grid,
             alpha=float(alpha), mask=int(mask), sets=int(sets))
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one analytic sky at low resolution, as an interactive user or a
        # sampler asks for it: 6.3 M samples, launch and call overhead count
        _case("analytic n32 host", "host", "fp64", "spiral", [32], 20.0, 20.0 / 512, [23.0]),
        # the smallest gridded pipeline (the tests' case): all latency
        _case("small grid host", "host", "fp64", "grid", [4, 8, 16], 30.0, 0.1, [1.4, 23.0],
              "32x32x32"),
        # a whole pipeline run (two frequencies, DM and FD) on 256^3 grids in
        # the default form, maps kept on the device
        _case("pipeline 256 fp64", "device", "fp64", "grid", [64, 128, 256], 30.0, 0.01,
              [1.4, 23.0], "256x256x256"),
        # the largest: Nside 1024, four shells, 512^3 grids, three frequencies
        _case("pipeline 512 fp64", "device", "fp64", "grid", [128, 256, 512, 1024], 30.0, 0.01,
              [0.408, 1.4, 30.0], "512x512x512"),
        # the same in the FP32-compensated form (the headline workload)
        _case("pipeline 512 fp32c", "device", "fp32c", "grid", [128, 256, 512, 1024], 30.0, 0.01,
              [0.408, 1.4, 30.0], "512x512x512"),
        # end to end from host FP32 grids to host maps, new grids every call
        _case("end to end 256 fp32c", "upload", "fp32c", "grid", [64, 128, 256], 30.0, 0.01,
              [1.4, 23.0], "256x256x256"),
        # JF12 with random fields on an odd, anisotropic grid, half of the sky
        # masked, CRE index away from 3, one frequency
        _case("jf12 masked fp64", "device", "fp64", "jf12", [32, 64, 128], 25.0, 0.02, [1.4],
              "199x201x67", alpha=2.7, mask=16),
        # gradient of a likelihood with respect to parameters and every voxel
        _case("gradient 256 fp64", "adjoint", "fp64", "grid", [64, 128, 256], 30.0, 0.01, [23.0],
              "256x256x256"),
        _case("gradient 256 fp32c", "adjoint", "fp32c", "grid", [64, 128, 256], 30.0, 0.01,
              [23.0], "256x256x256"),
        # a sampler's ensemble in one graph: parameter sets x three frequencies
        _case("ensemble fp32c", "batch", "fp32c", "grid", [64, 128, 256], 25.0, 0.01,
              [0.408, 1.4, 30.0], "256x256x256", sets=16),
        _case("ensemble fp64", "batch", "fp64", "grid", [32, 64], 20.0, 0.02, [1.4, 23.0],
              "96x96x48", sets=16),
        # one realisation of the turbulent fields, made on the device and seen
        _case("realisation 256 fp64", "generate", "fp64", "grid", [32, 64, 128], 30.0, 0.02,
              [30.0], "256x256x128"),
    ]


def _samples(c):
    """Reference loop iterations of one pass, and passes."""
    ns = [int(v) for v in c["nsides"].split(",")]
    o = workloads.make_obs(ns, c["r_max"], c["res"], freq_ghz=1.0)
    return workloads.samples_of(o), len(c["freqs"].split(","))


def _cost(c):
    """Rough relative time of a pass, to keep drawn cases under the largest."""
    s, p = _samples(c)
    w = 1.0 if c["form"] == "fp64" else 0.3
    w *= {"adjoint": 4.0, "batch": max(1, c["sets"])}.get(c["kind"], 1.0)
    nx, ny, nz = _dims(c)
    return s * p * w + 40.0 * nx * ny * nz * (c["kind"] in ("generate", "upload"))


def draw(rng):
    lu = lambda a, b: math.exp(rng.uniform(math.log(a), math.log(b)))  # noqa: E731
    kind, form = rng.choice([("host", "fp64"), ("device", "fp64"), ("device", "fp64"),
                             ("device", "fp32c"), ("upload", "fp32c"), ("adjoint", "fp64"),
                             ("adjoint", "fp32c"), ("batch", "fp32c"), ("batch", "fp64"),
                             ("generate", "fp64")])
    fields = "grid"
    if kind in ("host", "device"):
        fields = rng.choice(["spiral", "grid", "grid", "jf12"])
    top = {"host": 128, "device": 512, "upload": 256, "adjoint": 128, "batch": 128,
           "generate": 128}[kind]
    outer = 2 ** rng.randint(3, int(math.log2(top)))
    shells = rng.randint(1, 4)
    nsides = [max(2, outer >> (shells - 1 - k)) for k in range(shells)]
    big = {"generate": 200, "adjoint": 220, "upload": 220}.get(kind, 300)
    dims = [max(9, round(lu(16, big))) for _ in range(3)]
    freqs = sorted(rng.sample([0.408, 1.4, 4.76, 23.0, 30.0], 1 if kind in ("adjoint", "generate")
                              else rng.randint(1, 3)))
    res = lu(0.008, 0.1)
    alpha = rng.choice([3.0, 3.0, 2.7, 3.3])
    mask = rng.choice([0, 0, 8, 32]) if kind == "device" else 0
    c = _case(None, kind, form, fields, nsides, rng.uniform(8.0, 30.0), round(res, 5), freqs,
              "x".join(map(str, dims)) if fields != "spiral" else "", alpha, mask,
              rng.randint(3, 24) if kind == "batch" else 0)
    while _cost(c) > 4e10:
        c["res"] = round(c["res"] * 1.5, 5)
    return c


# ---- inputs ------------------------------------------------------------------

def _dims(c):
    return tuple(int(v) for v in c["grid"].split("x")) if c["grid"] else (0, 0, 0)


def _desc(c):
    d = workloads.grid_desc(2)
    d.nx, d.ny, d.nz = _dims(c)
    return d


def _noise(dims, seed, dtype):
    """Unit-variance Gaussian field with power spectrum k^-11/3."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(dims, generator=g, device="cuda", dtype=dtype)
    k = [torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=dtype) for n in dims[:2]]
    k.append(torch.fft.rfftfreq(dims[2], 1.0 / dims[2], device="cuda", dtype=dtype))
    kk = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    amp = torch.where(kk > 0, kk.clamp_min(1e-30) ** (-11.0 / 12.0), torch.zeros_like(kk))
    x = torch.fft.irfftn(torch.fft.rfftn(x) * amp, s=dims)
    x -= x.mean()
    return x / x.std()


def _grids(c, seed):
    """(bx, by, bz, ne) flat float64 tensors in CGS: 1 muG rms turbulence and a
    lognormal n_e of mean 0.03 cm^-3 (fluctuations of both signs around the
    analytic disk for the gradient).  FP32 numbers in the FP32C form."""
    dims = _dims(c)
    dt = torch.float64 if c["form"] == "fp64" else torch.float32
    b = [_noise(dims, seed * 16 + k, dt) * (U.muGauss / math.sqrt(3.0)) for k in range(3)]
    g = _noise(dims, seed * 16 + 3, dt)
    ne = 0.03 * torch.exp(0.5 * g - 0.125)
    if c["kind"] == "adjoint":
        ne = ne - 0.03
    return [t.to(dt).double().reshape(-1).contiguous() for t in (*b, ne)]


def _params(c, seed, count=1):
    """Regular-field parameters of `count` models, drawn like a sampler's."""
    r = np.random.Generator(np.random.PCG64(seed))
    return [dict(b0_muG=r.uniform(2, 8), pitch_deg=r.uniform(-40, -5), hb_kpc=r.uniform(0.5, 2))
            for _ in range(count)]


def _models(c, par):
    m = workloads.spiral_models(**par)
    m.cre_ana.alpha = c["alpha"]
    if c["fields"] == "spiral":
        return m
    m.brnd = abi.HXG_BRND_GRID
    if c["kind"] in ("adjoint", "generate"):
        m.ternd = abi.HXG_TERND_GRID    # fluctuations on the analytic disk
    else:
        m.tereg = abi.HXG_TEREG_GRID
    if c["fields"] == "jf12":
        m.breg = abi.HXG_BREG_JF12
        j = m.jf12
        for k, v in JF12.items():
            unit = (U.kpc if k in ("h_disk", "w_disk", "rn", "rs", "wh", "z0", "rpc_X", "r0_X")
                    else U.rad if k == "Xtheta" else U.muGauss)
            setattr(j, k, v * unit)
    return m


# JF12 best-fit values (Jansson & Farrar 2012, ApJ 757, 14): muG, kpc, degrees
JF12 = dict(b_arm1=0.1, b_arm2=3.0, b_arm3=-0.9, b_arm4=-0.8, b_arm5=-2.0, b_arm6=-4.2,
            b_arm7=0.0, b_ring=0.1, h_disk=0.40, w_disk=0.27, Bn=1.4, Bs=-1.1, rn=9.22,
            rs=16.7, wh=0.2, z0=5.3, B0_X=4.6, Xtheta=49.0, rpc_X=4.8, r0_X=2.9)


def _passes(c):
    ns = [int(v) for v in c["nsides"].split(",")]
    freqs = [float(v) for v in c["freqs"].split(",")]
    out = workloads.config_grid(ns, c["r_max"], c["res"], freqs)
    for o in out:
        o.do_mask = int(c["mask"] > 0)
    return out


def _mask(c, seed):
    r = np.random.Generator(np.random.PCG64(seed + 5))
    return (r.random(abi.npix(c["mask"])) > 0.5).astype(np.float64)


def _sizes(o):
    a, b, s = abi.obs_output_sizes(o)
    return (a, b, s, s, s)


def _device_maps(o):
    return [torch.zeros(n, dtype=torch.float64, device="cuda") if n else None for n in _sizes(o)]


def _turbulence(c):
    # break wavenumbers off the lattice of the box, where a rounding would decide
    es = abi.BrndEs(rms=0.8 * U.muGauss, k0=9.7, k1=0.11, a0=1.7, a1=0.0, rho=3.0,
                    r0=8 * U.kpc, z0=1 * U.kpc)
    dft = abi.TerndDft(rms=0.01, k0=0.06, a0=-11.0 / 3.0, r0=8 * U.kpc, z0=1 * U.kpc)
    return es, dft


def prepare(case, seed):
    c = case
    kind, form = c["kind"], c["form"]
    passes = _passes(c)
    par = _params(c, seed, max(1, c["sets"]))
    s = {"case": c, "passes": passes, "kind": kind}
    if kind == "adjoint":
        m = _models(c, par[0])
        p = torch.tensor(_params8(m), dtype=torch.float64, device="cuda", requires_grad=True)
        grids = [g.requires_grad_() for g in _grids(c, seed)]
        s.update(los=LOSMaps(passes[0], m, _desc(c), precision=form), params=p, grids=grids,
                 target=_targets(passes[0], seed))
        return s
    ig = Integrator(form)
    s["integ"] = ig
    ig.set_models(_models(c, par[0]))
    if kind == "upload":
        host = [g.float().cpu().pin_memory().numpy() for g in _grids(c, seed)]
        s["host"] = host
        s["maps"] = [{k: (torch.zeros(n, dtype=torch.float64).pin_memory().numpy() if n else None)
                      for k, n in zip(KEYS, _sizes(o))} for o in passes]
        return s
    if c["grid"] and kind != "generate":
        bx, by, bz, ne = _grids(c, seed)
        ig.upload_grid_device(abi.HXG_FIELD_BRND, _desc(c), [bx, by, bz])
        ig.upload_grid_device(abi.HXG_FIELD_TEREG, _desc(c), [ne])
        ig.sync()
    if c["mask"]:
        ig.set_mask(c["mask"], _mask(c, seed))
    if kind == "device":
        s["maps"] = [_device_maps(o) for o in passes]
    elif kind == "generate":
        s["maps"] = [_device_maps(o) for o in passes]
        s["seeds"] = (seed * 2 + 1, seed * 2 + 2)
    elif kind == "batch":
        # every map of a kind in one tensor, an entry's maps are slices of it
        total = {k: sum(_sizes(o)[j] for o in passes) * len(par) for j, k in enumerate(KEYS)}
        s["maps"] = {k: torch.zeros(n, dtype=torch.float64, device="cuda")
                     for k, n in total.items()}
        at, entries = dict.fromkeys(KEYS, 0), []
        for p in par:
            for o in passes:
                outs = {}
                for k, n in zip(KEYS, _sizes(o)):
                    if n:
                        outs[k] = s["maps"][k][at[k]:at[k] + n]
                        at[k] += n
                entries.append((_models(c, p), o, outs))
        s["batch"] = ig.batch(entries)
    return s


def _params8(m):
    return [m.spiral.b0, m.spiral.pitch, m.spiral.r_scale, m.spiral.h_scale, m.te_exp.n0,
            m.te_exp.r_scale, m.te_exp.h_scale, m.cre_ana.j0]


def _targets(o, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    return [torch.randn(n, generator=g, device="cuda", dtype=torch.float64) * w
            for n, w in zip(_sizes(o), LOSS_SCALE)]


def run(state):
    s = state
    kind = s["kind"]
    if kind == "host":
        return s["integ"].write_grid_multi(s["passes"])
    if kind == "upload":
        bx, by, bz, ne = s["host"]
        d = _desc(s["case"])
        s["integ"].upload_grid(abi.HXG_FIELD_BRND, d, [bx, by, bz])
        s["integ"].upload_grid(abi.HXG_FIELD_TEREG, d, [ne])
        return s["integ"].write_grid_multi(s["passes"], out=s["maps"])
    if kind == "adjoint":
        leaves = [s["params"], *s["grids"]]
        for t in leaves:
            t.grad = None
        maps = s["los"](s["params"], s["grids"][:3], s["grids"][3])
        loss = sum((((m - t) / w) ** 2).sum()
                   for m, t, w in zip(maps, s["target"], LOSS_SCALE))
        loss.backward()
        return {"maps": [m.detach() for m in maps], "grads": [t.grad for t in leaves]}
    if kind == "batch":
        s["batch"].run()
        return s["maps"]
    if kind == "generate":
        d, (es, dft) = _desc(s["case"]), _turbulence(s["case"])
        obs3 = [s["passes"][0].observer[k] for k in range(3)]
        s["integ"].generate_brnd_es(d, es, obs3, s["seeds"][0])
        s["integ"].generate_ternd_dft(d, dft, obs3, s["seeds"][1])
    s["integ"].write_grid_multi_device(list(zip(s["passes"], s["maps"])))
    return s["maps"]


def work(case):
    """The grid values and maps once, and per sample inside the cuts about 150
    flops of geometry, interpolation, models and emissivity plus 30 for each
    frequency's phase and sums (three times that for a gradient)."""
    c = case
    ns = [int(v) for v in c["nsides"].split(",")]
    passes = _passes(c)
    # samples inside the cuts, from the same shells at Nside <= 16
    o = workloads.make_obs([min(n, 16) for n in ns], c["r_max"], c["res"], freq_ghz=1.0)
    inside = sum(v * (n / min(n, 16)) ** 2 for v, n in zip(workloads.valid_samples(o), ns))
    if c["mask"]:
        inside *= 0.5
    nx, ny, nz = _dims(c)
    elem = 4 if c["form"] == "fp32c" else 8
    grid = nx * ny * nz * 4 * elem
    maps = sum(sum(_sizes(p)) for p in passes) * 8
    flops, nbytes = inside * (150 + 30 * len(passes)), grid + maps
    if c["kind"] == "adjoint":
        flops, nbytes = 3 * flops, 2 * nbytes + nx * ny * nz * 4 * 8
    elif c["kind"] == "batch":
        flops, nbytes = flops * c["sets"], grid + maps * c["sets"]
    elif c["kind"] == "generate":
        # 7 complex transforms and the deviates
        n = nx * ny * nz
        flops += n * (7 * 5 * math.log2(n) + 300)
        nbytes += n * 32
    return {"bytes": float(nbytes), "flops": float(flops)}


# ---- the same outputs in plain torch, 64 bits -----------------------------------
# CGS constants of the model definitions
PI = math.pi
KPC = 3.0856775806e21
QE, CL, KB, HP = 4.80320425e-10, 2.99792458e10, 1.380622e-16, 6.626075540e-27
MEC2 = 0.51099907e-3 * 1.60217733e-12 * 1e9
MEC = MEC2 / CL
GEV = 1.60217733e-12 * 1e9


def _ar(n):
    return torch.arange(n, device="cuda", dtype=torch.int64)


def _ring_angles(nside):
    """(theta, phi) of every RING pixel (Gorski et al. 2005, eqs. 4-9)."""
    p = _ar(12 * nside * nside)
    cap = 2 * nside * (nside - 1)
    z = torch.empty_like(p, dtype=torch.float64)
    s, phi = z.clone(), z.clone()

    def ring(q):                   # ring and index in it of a north-cap pixel
        i = (torch.sqrt((q + 1).double() / 2.0 + 0.25) + 0.5).long()
        i = torch.where(2 * i * (i - 1) > q, i - 1, i)
        i = torch.where(2 * i * (i + 1) <= q, i + 1, i)
        return i, q - 2 * i * (i - 1)
    for north in (True, False):
        at = p < cap if north else p >= p.numel() - cap
        q = p[at] if north else p.numel() - 1 - p[at]
        i, j = ring(q)
        t = (i * i).double() / (3.0 * nside * nside)
        z[at] = (1.0 - t) if north else (t - 1.0)
        s[at] = torch.sqrt(t * (2.0 - t))
        j = j if north else 4 * i - 1 - j
        phi[at] = (j.double() + 0.5) * (0.5 * PI) / i.double()
    at = (p >= cap) & (p < p.numel() - cap)
    q = p[at] - cap
    i = torch.div(q, 4 * nside, rounding_mode="floor") + nside
    j = q % (4 * nside)
    half = 0.5 * ((i - nside) % 2 == 0).double()
    z[at] = (2 * nside - i).double() * (2.0 / (3.0 * nside))
    s[at] = torch.sqrt((1.0 - z[at]) * (1.0 + z[at]))
    phi[at] = (j.double() + half) * (0.5 * PI / nside)
    return torch.atan2(s, z), phi


def _ring_info(nside, r):
    """First pixel, length, colatitude and phase shift of rings r (1..4n-1)."""
    n = torch.where(r > 2 * nside, 4 * nside - r, r)
    cap = n < nside
    t = (n * n).double() / (3.0 * nside * nside)
    zc, ze = 1.0 - t, (2 * nside - n).double() * (2.0 / (3.0 * nside))
    th = torch.where(cap, torch.atan2(torch.sqrt(t * (2.0 - t)), zc),
                     torch.acos(ze.clamp(-1, 1)))
    length = torch.where(cap, 4 * n, torch.full_like(n, 4 * nside))
    start = torch.where(cap, 2 * n * (n - 1),
                        2 * nside * (nside - 1) + (n - nside) * 4 * nside)
    shift = torch.where(cap, torch.ones_like(t), ((n - nside) % 2 == 0).double())
    south = n != r
    return (torch.where(south, 12 * nside * nside - start - length, start), length,
            torch.where(south, PI - th, th), shift)


def _interp(nside, theta, phi):
    """The 4 pixels and weights of the HEALPix bilinear interpolation."""
    z = torch.cos(theta)
    az = z.abs()
    cap = (nside * torch.sqrt(3.0 * (1.0 - az))).long()
    r1 = torch.where(az <= 2.0 / 3.0, (nside * (2.0 - 1.5 * z)).long(),
                     torch.where(z > 0, cap, 4 * nside - cap - 1))
    r2 = r1 + 1
    pix, wgt, th = [], [], []
    for r in (r1, r2):
        start, length, t, shift = _ring_info(nside, r.clamp(1, 4 * nside - 1))
        dphi = 2.0 * PI / length.double()
        x = phi / dphi - 0.5 * shift
        i = torch.floor(x)
        w = x - i
        i = i.long()
        pix += [start + i % length, start + (i + 1) % length]
        wgt += [1.0 - w, w]
        th.append(t)
    top, bot = r1 == 0, r2 == 4 * nside
    t1 = torch.where(top, torch.zeros_like(theta), th[0])
    t2 = torch.where(bot, torch.full_like(theta, PI), th[1])
    f = (theta - t1) / (t2 - t1)
    # beyond the first / last ring the pole is the mean of that ring's 4 pixels
    w1 = [torch.where(top, 0.25 * (1 - f), w * (1 - f)) for w in wgt[:2]]
    w2 = [torch.where(bot, 0.25 * f, w * f) for w in wgt[2:]]
    w2 = [torch.where(top, w + 0.25 * (1 - f), w) for w in w2]
    w1 = [torch.where(bot, w + 0.25 * f, w) for w in w1]
    npx = 12 * nside * nside
    p1 = [torch.where(top, (q + 2) % 4, p) for p, q in zip(pix[:2], pix[2:])]
    p2 = [torch.where(bot, (p + 2 - (npx - 4)) % 4 + npx - 4, q)
          for p, q in zip(pix[:2], pix[2:])]
    return torch.stack(p1 + p2), torch.stack(w1 + w2)


def _nest_to_ring(nside):
    """RING index of every NESTED pixel."""
    k = int(math.log2(nside))
    q = _ar(12 * nside * nside)
    face, q = q >> (2 * k), q & (nside * nside - 1)
    ix, iy = torch.zeros_like(q), torch.zeros_like(q)
    for b in range(k):
        ix |= ((q >> (2 * b)) & 1) << b
        iy |= ((q >> (2 * b + 1)) & 1) << b
    jr = (2 + (face >> 2)) * nside - ix - iy - 1
    north, south = jr < nside, jr > 3 * nside
    nr = torch.where(north, jr, torch.where(south, 4 * nside - jr, torch.full_like(jr, nside)))
    before = torch.where(north, 2 * jr * (jr - 1),
                         torch.where(south, 12 * nside * nside - 2 * nr * (nr + 1),
                                     2 * nside * (nside - 1) + (jr - nside) * 4 * nside))
    kshift = torch.where(north | south, torch.zeros_like(jr), (jr - nside) & 1)
    jpll = ((face & 3) << 1) + 1 - ((face >> 2) & 1)
    jp = torch.div(jpll * nr + ix - iy + 1 + kshift, 2, rounding_mode="trunc")
    jp = torch.where(jp < 1, jp + 4 * nside, torch.where(jp > 4 * nside, jp - 4 * nside, jp))
    return before + jp - 1


def _mask_at(mask, nside_mask, nside):
    """The sky mask at another Nside: parent of a pixel, or any of its children."""
    m = torch.as_tensor(mask, device="cuda")[_nest_to_ring(nside_mask)] > 0
    if nside >= nside_mask:
        m = m.repeat_interleave((nside // nside_mask) ** 2)
    else:
        m = m.reshape(12 * nside * nside, -1).any(1)
    out = torch.empty_like(m)
    out[_nest_to_ring(nside)] = m
    return out


def _b_jf12(x, y, z):
    p = JF12
    r, phi = torch.sqrt(x * x + y * y), torch.atan2(y, x)
    az, rho = z.abs(), torch.sqrt(x * x + y * y + z * z)
    zp = 1.0 / (1.0 + torch.exp(-2.0 / p["w_disk"] * (az - p["h_disk"])))
    f = [0.130, 0.165, 0.094, 0.122, 0.13, 0.118, 0.084, 0.156]
    rc = [5.1, 6.3, 7.1, 8.3, 9.8, 11.4, 12.7, 15.5]
    bv = [p["b_arm%d" % k] for k in range(1, 8)]
    bv.append(-sum(a * b for a, b in zip(f, bv)) / f[7])
    inc = math.radians(11.5)
    ct = 1.0 / math.tan(math.radians(90.0 - 11.5))
    rn = r * torch.exp(-ct * (phi - PI))
    rn = torch.where(rn > rc[7], r * torch.exp(-ct * (phi + PI)), rn)
    rn = torch.where(rn > rc[7], r * torch.exp(-ct * (phi + 3 * PI)), rn)
    arm = torch.zeros_like(r)
    for k in range(7, -1, -1):
        arm = torch.where(rn < rc[k], torch.full_like(r, bv[k]), arm)
    b0 = (5.0 / r) * (1.0 - zp)
    disk = r >= 5.0
    ring = (r > 3.0) & ~disk
    zero = torch.zeros_like(r)
    br = torch.where(disk, arm * b0 * math.sin(inc), zero)
    bp = torch.where(disk, arm * b0 * math.cos(inc),
                     torch.where(ring, b0 * p["b_ring"], zero))
    up = z >= 0
    b1 = torch.where(up, torch.full_like(r, p["Bn"]), torch.full_like(r, p["Bs"]))
    rh = torch.where(up, torch.full_like(r, p["rn"]), torch.full_like(r, p["rs"]))
    bp = bp + zp * b1 * (1.0 - 1.0 / (1.0 + torch.exp(-2.0 / p["wh"] * (r - rh)))) \
        * torch.exp(-az / p["z0"])
    tx = math.tan(math.radians(p["Xtheta"]))
    rcx = p["rpc_X"] + az / tx
    inner = r < rcx
    q = p["rpc_X"] / rcx
    rp = torch.where(inner, r * q, r - az / tx)
    bx = p["B0_X"] * torch.where(inner, q * q, rp / r) * torch.exp(-rp / p["r0_X"])
    ang = torch.where(inner, torch.atan2(az, r - rp),
                      torch.full_like(r, math.radians(p["Xtheta"])))
    br = br + bx * torch.cos(ang) * torch.where(z < 0, -1.0, 1.0)
    bz = bx * torch.sin(ang)
    out = (r > 20.0) | (rho < 1.0)
    c, s = x / r, y / r
    return [torch.where(out, torch.full_like(r, 1e-12), v * 1e-6)
            for v in (br * c - bp * s, br * s + bp * c, bz)]


class _Sky:
    """The line-of-sight integral of one parameter set over all passes."""

    def __init__(self, c, passes, par8, rec, mask=None):
        self.c, self.passes, self.par, self.rec, self.mask = c, passes, par8, rec, mask
        o = passes[0]
        self.obs = [o.observer[k] for k in range(3)]
        self.shells = [(o.nside_shell[s], o.radii_shell[s], o.radii_shell[s + 1])
                       for s in range(o.total_shell)]
        self.res, self.rmax, self.zmax = o.oc_r_res, o.gc_r_max, o.gc_z_max
        self.grid_ne_only = c["fields"] != "spiral" and c["kind"] not in ("adjoint", "generate")

    def fields(self, x, y, z):
        b0, pitch, rs, hs, n0, rn, hn, _ = self.par
        r2 = x * x + y * y
        r = torch.sqrt(r2)
        if self.c["fields"] == "jf12":
            b = _b_jf12(x / KPC, y / KPC, z / KPC)
        else:
            rsun = math.hypot(self.obs[0], self.obs[1])
            on = (r <= 20 * KPC) & (r >= 3 * KPC)
            amp = torch.where(on, b0 * torch.exp(-(r - rsun) / rs - z.abs() / hs),
                              torch.zeros_like(r)) / r
            sp, cp = torch.sin(pitch), torch.cos(pitch)
            b = [amp * (sp * x - cp * y), amp * (sp * y + cp * x), torch.zeros_like(r)]
        ne = torch.zeros_like(r)
        if not self.grid_ne_only:
            ne = n0 * torch.exp(-r / rn - z.abs() / hn)
        if self.rec is not None:
            g = self.trilinear(x, y, z)
            b = [v + g[..., k] for k, v in enumerate(b)]
            ne = ne + g[..., 3]
        return b, ne.clamp_min(0.0), r

    def trilinear(self, x, y, z):
        dims = _dims(self.c)
        box = [v * KPC for v in workloads.BOX_KPC]
        inside, cell, frac = None, [], []
        for k, (p, n) in enumerate(zip((x, y, z), dims)):
            t = (p - box[2 * k]) * ((n - 1) / (box[2 * k + 1] - box[2 * k]))
            ok = (t > 0) & (t < n - 1)
            inside = ok if inside is None else inside & ok
            i = torch.floor(t).clamp(0, n - 2)
            cell.append(i.long())
            frac.append(t - i)
        at = torch.nonzero(inside.reshape(-1)).reshape(-1)
        i, j, k = (v.reshape(-1)[at] for v in cell)
        f = [v.reshape(-1)[at][:, None] for v in frac]
        base = (i * dims[1] + j) * dims[2] + k
        sx, sy = dims[1] * dims[2], dims[2]
        val = None
        for dx in (0, 1):
            for dy in (0, 1):
                for dz in (0, 1):
                    w = (f[0] if dx else 1 - f[0]) * (f[1] if dy else 1 - f[1]) \
                        * (f[2] if dz else 1 - f[2])
                    t = self.rec.index_select(0, base + dx * sx + dy * sy + dz) * w
                    val = t if val is None else val + t
        out = torch.zeros((inside.numel(), 4), dtype=torch.float64, device="cuda")
        return out.index_copy(0, at, val).reshape(*inside.shape, 4)

    def rays(self, s, pix, theta, phi, inner):
        """Per-pixel sums of shell s: dm, fd and [I, Q, U] of every pass, before
        the merges; inner: the Faraday depth of the shells before it."""
        _, d0, d1 = self.shells[s]
        steps = math.floor(d1 / self.res - d0 / self.res)
        dl = (d1 - d0) / steps
        th, ph = theta[pix], phi[pix]
        st, ct, sp, cp = torch.sin(th), torch.cos(th), torch.sin(ph), torch.cos(ph)
        u = (cp * st, sp * st, ct)
        # the steps any of these rays can have inside the cuts
        ou = sum(a * b for a, b in zip(self.obs, u))
        far = -ou + torch.sqrt((ou * ou + self.rmax ** 2 -
                                sum(a * a for a in self.obs)).clamp_min(0))
        far = torch.minimum(far, (self.zmax + abs(self.obs[2])) / ct.abs().clamp_min(1e-9))
        last = min(steps, int((far.max().item() - d0) / dl) + 2)
        if last < 1:
            last = 1
        d = d0 + (torch.arange(last, device="cuda", dtype=torch.float64) + 0.5) * dl
        col = lambda v: v[:, None]  # noqa: E731
        x, y, z = (col(a) * d + o for a, o in zip(u, self.obs))
        on = (x * x + y * y + z * z <= self.rmax ** 2) & (z.abs() <= self.zmax)
        (bx, by, bz), ne, r = self.fields(x, y, z)
        zero = torch.zeros_like(x)
        ne = torch.where(on, ne, zero)
        dm = ne.sum(1) * dl
        bpar = bx * col(u[0]) + by * col(u[1]) + bz * col(u[2])
        run = torch.cumsum(ne * bpar, 1) * (-(QE ** 3) / (2 * PI * MEC2 ** 2) * dl)
        fd = run[:, -1]
        xv = col(sp) * bx - col(cp) * by
        yv = col(st) * bz - col(ct) * (col(cp) * bx + col(sp) * by)
        b2 = xv * xv + yv * yv
        alpha, R0 = self.c["alpha"], math.hypot(self.obs[0], self.obs[1])
        prof = torch.exp((R0 - r) / (5 * KPC)) / torch.cosh(z / KPC) ** 2
        gam0 = 20.6 * GEV / MEC2
        unit = 4 * PI * MEC / (GEV * 1e4 * math.sqrt(1 - 1 / gam0))
        n0u = gam0 ** alpha * unit
        e = 0.5 * (1.0 - alpha)
        gt = math.gamma(0.25 * alpha + 19 / 12) * math.gamma(0.25 * alpha - 1 / 12)
        gp = math.gamma(0.25 * alpha + 7 / 12) * math.gamma(0.25 * alpha - 1 / 12)
        # |B_perp|^(1 - e), with the angle's factors 1 / |B_perp|^2
        ok = on & (b2 > 0)
        b2s = torch.where(ok, b2, torch.ones_like(b2))
        wt = torch.where(ok, prof * b2s ** (0.5 * (1 - e)), zero)
        wq = wt / b2s
        c2, s2 = (xv * xv - yv * yv) * wq, 2 * xv * yv * wq
        j0 = self.par[7]
        stokes = []
        for o in self.passes:
            nu = o.sync_freq
            l2, i2bt = (CL / nu) ** 2, CL ** 2 / (2 * KB * nu * nu)
            q = HP * nu / (KB * 2.725)
            tc = (math.exp(q) - 1) ** 2 / (q * q * math.exp(q))
            a = (2 * PI * nu * MEC / (3 * QE)) ** e
            k = n0u * 1.73205081 * QE ** 3 * a * dl * i2bt * tc
            kt = j0 * (k * gt / (4 * PI * MEC2 * (1 + alpha)))
            kp = j0 * (k * gp / (16 * PI * MEC2))
            ang = 2 * l2 * (run + col(inner)) if o.do_fd else 2 * l2 * run
            cf, sf = torch.cos(ang), torch.sin(ang)
            stokes.append([wt.sum(1) * kt, (cf * c2 - sf * s2).sum(1) * kp,
                           (sf * c2 + cf * s2).sum(1) * kp])
        return dm, fd, stokes

    def chunks(self, s, size):
        nside, d0, d1 = self.shells[s]
        pix = _ar(12 * nside * nside)
        if self.mask is not None:
            pix = pix[_mask_at(*self.mask, nside)]
        n = max(1, int(size / max(1, (d1 - d0) / self.res)))
        return pix.split(n) if pix.numel() else []

    def inner(self, nside, theta, phi, fd, pix):
        if not self.passes[0].do_fd:
            return torch.zeros(pix.numel(), dtype=torch.float64, device="cuda")
        p, w = _interp(self.passes[0].nside_fd, theta[pix], phi[pix])
        return (fd[p] * w).sum(0)

    def maps(self):
        """The maps of every pass, as the API lays them out; keeps the FD map
        that each shell reads."""
        outs = [[torch.zeros(n, dtype=torch.float64, device="cuda") if n else None
                 for n in _sizes(o)] for o in self.passes]
        fd_out = outs[0][1] if outs[0][1] is not None else torch.zeros(12, device="cuda",
                                                                       dtype=torch.float64)
        self.fd_before = []
        for s, (nside, _, _) in enumerate(self.shells):
            theta, phi = _ring_angles(nside)
            self.fd_before.append(fd_out.clone())
            part = [torch.zeros(12 * nside * nside, dtype=torch.float64, device="cuda")
                    for _ in range(2 + 3 * len(self.passes))]
            for pix in self.chunks(s, 6e6):
                dm, fd, st = self.rays(s, pix, theta, phi,
                                       self.inner(nside, theta, phi, fd_out, pix))
                for t, v in zip(part, [dm, fd] + [x for row in st for x in row]):
                    t[pix] = v
            for k, out in enumerate(outs):
                src = part[:2] + part[2 + 3 * k:5 + 3 * k]
                for t, v in zip(out, src):
                    if t is not None:
                        t += self.merged(v, nside, t.numel())
        return outs

    @staticmethod
    def merged(v, nside, npix):
        n = int(round(math.sqrt(npix / 12)))
        if n == nside:
            return v
        p, w = _interp(nside, *_ring_angles(n))
        return (v[p] * w).sum(0)

    def gradients(self, g):
        """dL/d(parameters, records) from dL/d(maps) of the one pass: the shells
        from the outermost in, the inner Faraday depth's share added to dL/dFD."""
        gp, gr = torch.zeros_like(self.par), torch.zeros_like(self.rec)
        gfd = g[1].clone()
        n_out = int(round(math.sqrt(gfd.numel() / 12)))
        for s in range(len(self.shells) - 1, -1, -1):
            nside = self.shells[s][0]
            theta, phi = _ring_angles(nside)
            up = []
            for v in (g[0], gfd, g[2], g[3], g[4]):
                if nside == n_out:
                    up.append(v.clone())
                    continue
                p, w = _interp(nside, *_ring_angles(n_out))
                t = torch.zeros(12 * nside * nside, dtype=torch.float64, device="cuda")
                up.append(t.index_add(0, p.reshape(-1), (w * v).reshape(-1)))
            add = torch.zeros_like(gfd)
            for pix in self.chunks(s, 3e6):
                inner = self.inner(nside, theta, phi, self.fd_before[s], pix).requires_grad_()
                self.par.requires_grad_()
                self.rec.requires_grad_()
                dm, fd, st = self.rays(s, pix, theta, phi, inner)
                got = torch.autograd.grad([dm, fd, *st[0]], [self.par, self.rec, inner],
                                          [t[pix] for t in up])
                gp += got[0]
                gr += got[1]
                p, w = _interp(n_out, theta[pix], phi[pix])
                add.index_add_(0, p.reshape(-1), (w * got[2]).reshape(-1))
            self.par.requires_grad_(False)
            self.rec.requires_grad_(False)
            gfd = gfd + add
        return gp, gr


def _philox(seed, n, block):
    """Philox4x32-10 of counters {cell, 0, block, tag}: two 53-bit uniforms."""
    c = [_ar(n), torch.zeros_like(_ar(n)), torch.full_like(_ar(n), block),
         torch.full_like(_ar(n), 0x52464721)]
    k, low = [seed & 0xFFFFFFFF, seed >> 32], 0xFFFFFFFF

    def mul(m, a):
        t = a * (m & 0xFFFF)
        v = a * (m >> 16) + (t >> 16)
        return v >> 16, ((v & 0xFFFF) << 16) | (t & 0xFFFF)
    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k[0], l1, h0 ^ c[3] ^ k[1], l0]
        k = [(k[0] + 0x9E3779B9) & low, (k[1] + 0xBB67AE85) & low]
    return [((((c[2 * q] << 21) ^ (c[2 * q + 1] >> 11)) & ((1 << 53) - 1)).double() + 0.5)
            * 2.0 ** -53 for q in (0, 1)]


def _normals(seed, n, block):
    u, v = _philox(seed, n, block)
    r = torch.sqrt(-2.0 * torch.log(u))
    return torch.complex(r * torch.cos(2 * PI * v), r * torch.sin(2 * PI * v))


def _exact_turbulence(c, sky, seeds):
    """Records of the generated fields: Fourier-space Gaussian fields with the
    template's spectra, the profile and anisotropy along the regular field,
    and the divergence-free projection."""
    dims = _dims(c)
    n = dims[0] * dims[1] * dims[2]
    box = [v * KPC for v in workloads.BOX_KPC]
    size = [box[2 * k + 1] - box[2 * k] for k in range(3)]
    ks, xs = [], []
    for k in range(3):
        i = torch.arange(dims[k], device="cuda", dtype=torch.float64)
        ks.append((i - dims[k] * (i >= (dims[k] + 1) // 2)) * (KPC / size[k]))
        xs.append(i * size[k] / (dims[k] - 1) + box[2 * k])
    kv = torch.meshgrid(*ks, indexing="ij")
    x, y, z = torch.meshgrid(*xs, indexing="ij")
    kk = sum(v * v for v in kv)
    km = torch.sqrt(kk)
    dk3 = KPC ** 3 / (size[0] * size[1] * size[2])
    ifft = lambda v: torch.fft.ifftn(v, norm="forward")  # noqa: E731

    def var(v):                     # over the first n of the 2 n real numbers
        t = torch.view_as_real(v.reshape(-1)).reshape(-1)[:n]
        return ((t - t.mean()) ** 2).mean()
    rc = torch.sqrt(x * x + y * y) - abs(sky.obs[0])
    prof = torch.exp(-0.5 * (rc / (8 * KPC) + (z.abs() - abs(sky.obs[2])) / KPC))
    ks_ = torch.where(kk > 0, km, torch.ones_like(km))
    # n_e: k^-11/3 above k0
    spec = torch.where(ks_ >= 0.06, 0.01 * (ks_ / 0.06) ** (-11.0 / 3.0) / (4 * PI * ks_ ** 2),
                       torch.zeros_like(km))
    spec = torch.where(kk > 0, spec, torch.zeros_like(km))
    f = ifft(_normals(seeds[1], n, 0).reshape(dims) * torch.sqrt(spec * dk3))
    ne = f.real * prof * (0.01 / torch.sqrt(var(f)))
    # B: k^6 below k1, k^-a1 to k0, k^-a0 above
    rms, k0, k1, a0, a1, rho = 0.8e-6, 9.7, 0.11, 1.7, 0.0, 3.0
    spec = torch.where(ks_ < k1, (k0 / k1) ** a1 * (ks_ / k1) ** 6,
                       torch.where((ks_ > k1) & (ks_ < k0), (ks_ / k0) ** -a1,
                                   torch.where(ks_ > k0, (ks_ / k0) ** -a0,
                                               torch.zeros_like(km))))
    spec = torch.where(kk > 0, spec * rms ** 2 / (4 * PI * ks_ ** 2), torch.zeros_like(km))
    sig = torch.sqrt(spec * (dk3 / 3.0))
    c0 = ifft(_normals(seeds[0], n, 0).reshape(dims) * sig)
    c1 = ifft(_normals(seeds[0], n, 1).reshape(dims) * sig)
    ratio = prof * (rms / torch.sqrt(3.0 * var(c0)))
    b = [v * ratio for v in (c0.real, c0.imag, c1.imag)]
    (hx, hy, hz), _, _ = sky.fields(x, y, z)
    hh = torch.sqrt(hx * hx + hy * hy + hz * hz)
    none = hh == 0
    h = [v / torch.where(none, torch.ones_like(hh), hh) for v in (hx, hy, hz)]
    hb = sum(p * q for p, q in zip(h, b))
    norm = 1.0 / math.sqrt(rho * rho / 3.0 + 2.0 / 3.0 / (rho * rho))
    keep = (c0.real, c1.real, c1.imag)
    b = [torch.where(none, t, (p * hb * rho + (q - p * hb) / rho) * norm)
         for t, p, q in zip(keep, h, b)]
    even = lambda t: 0.5 * (t + torch.roll(t.flip((0, 1, 2)), (1, 1, 1), (0, 1, 2)))  # noqa: E731
    f = [even(torch.fft.fftn(t).real) for t in b]
    kb = sum(p * q for p, q in zip(kv, f))
    same = (kk == 0) | (f[0] ** 2 + f[1] ** 2 + f[2] ** 2 == 0)
    f = [math.sqrt(2.0) * torch.where(same, t, math.sqrt(3.0) * (t - p * kb / kk))
         for t, p in zip(f, kv)]
    out = [even(torch.fft.ifftn(t.to(torch.complex128)).real) for t in f]
    return torch.stack([t.reshape(-1) for t in (*out, ne)], 1)


def exact(case, seed):
    c = case
    samples, npass = _samples(c)
    if c["kind"] == "adjoint" and samples > 2e9:
        return None
    passes = _passes(c)
    par = _params(c, seed, max(1, c["sets"]))
    rec = None
    if c["grid"] and c["kind"] != "generate":
        rec = torch.stack(_grids(c, seed), 1)
    mask = (_mask(c, seed), c["mask"]) if c["mask"] else None
    skies = [_Sky(c, passes, torch.tensor(_params8(_models(c, p)), dtype=torch.float64,
                                          device="cuda"), rec, mask) for p in par]
    if c["kind"] == "generate":
        skies[0].rec = _exact_turbulence(c, skies[0], (seed * 2 + 1, seed * 2 + 2))
    if c["kind"] == "batch":
        got = [s.maps() for s in skies]
        return {k: torch.cat([row[j] for one in got for row in one if row[j] is not None])
                for j, k in enumerate(KEYS)}
    maps = skies[0].maps()
    if c["kind"] == "adjoint":
        g = [2 * (m - t) / w ** 2 for m, t, w in zip(maps[0], _targets(passes[0], seed),
                                                     LOSS_SCALE)]
        gp, gr = skies[0].gradients(g)
        return {"maps": maps[0], "grads": [gp, *gr.t().contiguous()]}
    if c["kind"] in ("host", "upload"):
        return [dict(zip(KEYS, row)) for row in maps]
    return maps
