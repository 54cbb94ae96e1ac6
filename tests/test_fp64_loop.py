"""The FP64 sample loop at its edges, against the CPU oracle (the reference's
operation order): windows trimmed by the cuts and cut into chunks, an inner
radius, the emissivity's power forms, exponents beyond the loops' own range,
grids of unequal odd axes, the observer outside the box, and caller-packed
records aligned to 16 bytes.  Bounds: those of the parity suite, 1e-10 of the
map maximum for DM and FD, 1e-9 for I, Q, U."""
import numpy as np
import pytest

from conftest import rel_err
from hammurabix_b200 import abi, workloads as W
from hammurabix_b200 import units as U

pytestmark = pytest.mark.gpu
KEYS = ("dm", "fd", "is", "qs", "us")


def _grids(dims, box=W.BOX_KPC, seed=3):
    r = np.random.Generator(np.random.PCG64(seed))
    d = W.grid_desc(2, box)
    d.nx, d.ny, d.nz = dims
    n = int(np.prod(dims))
    b = [1e-6 * r.standard_normal(n) for _ in range(3)]
    return {abi.HXG_FIELD_BRND: (d, b), abi.HXG_FIELD_TEREG: (d, [0.03 * (r.random(n) - 0.2)])}


def _models(gridded, **kw):
    m = W.grid_models() if gridded else W.spiral_models()
    m.cre_ana.alpha = kw.get("alpha", 3.0)
    m.cre_ana.beta = kw.get("beta", 0.0)
    m.breg = kw.get("breg", m.breg)
    m.spiral.h_scale = kw.get("hs", 1.0) * U.kpc
    m.cre = kw.get("cre", m.cre)
    m.cre_unif.alpha, m.cre_unif.E0, m.cre_unif.j0 = 3.0, 20.6 * U.GeV, 0.0217
    m.cre_unif.r0 = 6.0 * U.kpc
    m.lsa.b0, m.lsa.psi0, m.lsa.psi1, m.lsa.chi0 = (3e-6, 0.5, 0.02, 0.4)
    return m


CASES = {
    "one step per chunk": dict(nsides=[2, 4], res=1.3, grid=(9, 8, 5)),
    "few rays": dict(nsides=[1, 2, 8], res=0.05, grid=(17, 40, 11)),
    "many rays": dict(nsides=[16, 64], res=0.1, grid=(21, 19, 33)),
    "analytic": dict(nsides=[8, 16], res=0.05, grid=None),
    "inner radius": dict(nsides=[8, 16], res=0.05, grid=(21, 19, 33), r_min=7.0),
    "inner radius, analytic": dict(nsides=[8], res=0.05, grid=None, r_min=7.0),
    "index 2.5": dict(nsides=[8, 16], res=0.05, grid=(21, 19, 33), alpha=2.5),
    "index 1": dict(nsides=[8], res=0.05, grid=(21, 19, 33), alpha=1.0),
    "varying index": dict(nsides=[8], res=0.05, grid=(21, 19, 33), beta=0.05),
    "thin disk": dict(nsides=[8], res=0.05, grid=(21, 19, 33), hs=0.01),
    "uniform cre": dict(nsides=[8], res=0.05, grid=(21, 19, 33), cre=abi.HXG_CRE_UNIF),
    "lsa": dict(nsides=[8], res=0.05, grid=(21, 19, 33), breg=abi.HXG_BREG_LSA),
    "box beside the observer": dict(nsides=[8, 16], res=0.05, grid=(12, 15, 9),
                                    box=(-3.0, 12.0, -4.0, 9.0, 0.5, 4.0)),
    "observer off the plane": dict(nsides=[8, 16], res=0.05, grid=(12, 15, 9),
                                   observer=(0.0, 0.0, 11.0)),
    "outside the cuts": dict(nsides=[4], res=0.05, grid=(12, 15, 9),
                             observer=(60.0, 0.0, 0.0)),
}


@pytest.mark.parametrize("freq", [23.0, 0.408])
@pytest.mark.parametrize("name", list(CASES))
def test_fp64_loop_vs_oracle(oracle, name, freq):
    from hammurabix_b200.integrator import Integrator
    c = CASES[name]
    o = W.make_obs(c["nsides"], 22.0, c["res"], freq_ghz=freq,
                   observer_kpc=c.get("observer", W.OBSERVER_KPC))
    o.gc_r_min = c.get("r_min", 0.0) * U.kpc
    g = _grids(c["grid"], c.get("box", W.BOX_KPC)) if c["grid"] else None
    m = _models(c["grid"], **c)
    ref = oracle.write_grid(o, m, g)
    with Integrator("fp64") as ig:
        ig.set_models(m)
        for slot, (d, comps) in (g or {}).items():
            ig.upload_grid(slot, d, comps)
        got = ig.write_grid(o)
    for k in KEYS:
        if not np.abs(ref[k]).max() > 0:
            assert np.abs(got[k]).max() == 0, k
            continue
        assert rel_err(got[k], ref[k]) <= (1e-10 if k in ("dm", "fd") else 1e-9), k


@pytest.mark.parametrize("offset", [0, 2])
def test_noalloc_records_aligned_to_16_bytes(oracle, offset):
    """hxg_write_grid_noalloc on records `offset` doubles past a 32-byte line."""
    import ctypes as C

    import torch
    from hammurabix_b200 import _lib
    lib = _lib.load()
    o = W.make_obs([4, 8], 20.0, 0.1, freq_ghz=1.4)
    g = _grids((9, 11, 7))
    m = _models(True)
    d, b = g[abi.HXG_FIELD_BRND]
    rec = np.stack([*b, g[abi.HXG_FIELD_TEREG][1][0]], axis=1).reshape(-1)
    buf = torch.zeros(rec.size + 8, dtype=torch.float64, device="cuda")
    buf[offset:offset + rec.size] = torch.from_numpy(rec)
    npx = abi.npix(8)
    outs = [torch.zeros(npx, dtype=torch.float64, device="cuda") for _ in range(5)]
    st = torch.cuda.current_stream()
    _lib.check(lib.hxg_write_grid_noalloc(
        C.byref(o), C.byref(m), C.byref(d), C.c_void_p(buf.data_ptr() + 8 * offset),
        *(C.c_void_p(t.data_ptr()) for t in outs), C.c_void_p(st.cuda_stream)))
    torch.cuda.synchronize()
    ref = oracle.write_grid(o, m, g)
    for k, t in zip(KEYS, outs):
        assert rel_err(t.cpu().numpy(), ref[k]) <= (1e-10 if k in ("dm", "fd") else 1e-9), k
