"""Batches whose small parameter sets share kernels: groups of one instantiation (sets
with and without JF12, 1 to 3 passes, beside large sets), the kernels a run launches,
and which launch shapes tuning times.  Every entry against the same pass run alone: 1e-10
of the map maximum in FP64 (chunked sums of a few thousand terms), 1e-5 in FP32C."""
import numpy as np
import pytest

from conftest import rel_err
from hammurabix_b200 import abi, units as U, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
KEYS = ("dm", "fd", "is", "qs", "us")


def _integ(form, fields32):
    from hammurabix_b200.integrator import Integrator
    ig = Integrator(form)
    f = [torch.tensor(np.asarray(a, dtype=np.float64).reshape(-1), device="cuda")
         for a in fields32]
    ig.set_models(W.grid_models())
    ig.upload_grid_device(abi.HXG_FIELD_BRND, W.grid_desc(32), f[:3])
    ig.upload_grid_device(abi.HXG_FIELD_TEREG, W.grid_desc(32), f[3:])
    return ig


def _model(rng, kind):
    m = W.grid_models(W.spiral_models(b0_muG=rng.uniform(2, 8), pitch_deg=rng.uniform(-40, -5)))
    if kind == "jf12":
        m.breg = abi.HXG_BREG_JF12
        for k, v in dict(b_arm2=3.0, b_arm5=-2.0, b_ring=0.1, Bn=1.4, Bs=-1.1, B0_X=4.6).items():
            setattr(m.jf12, k, v * U.muGauss)
        for k, v in dict(h_disk=0.4, w_disk=0.27, rn=9.22, rs=16.7, wh=0.2, z0=5.3, rpc_X=4.8,
                         r0_X=2.9).items():
            setattr(m.jf12, k, v * U.kpc)
        m.jf12.Xtheta = 49.0 * U.rad
    elif kind == "thin":                # exponents beyond the unchecked range
        m.spiral.h_scale = 0.01 * U.kpc
    elif kind == "index":
        m.cre_ana.beta = 0.02
    return m


def _entries(rng, sets):
    """sets: (model, Nsides, frequencies) each."""
    out = []
    for kind, nsides, freqs in sets:
        m = _model(rng, kind)
        for o in W.config_grid(nsides, 20.0, 0.1, freqs):
            n = abi.obs_output_sizes(o)
            out.append((m, o, {k: torch.full((c,), np.nan, dtype=torch.float64, device="cuda")
                               for k, c in zip(KEYS, (n[0], n[1], n[2], n[2], n[2])) if c}))
    return out


def _check(ig, entries, which, tol):
    for k in which:
        m, o, outs = entries[k]
        one = {q: torch.zeros_like(t) for q, t in outs.items()}
        ig.set_models(m)
        ig.write_grid_device(o, *(one.get(q) for q in KEYS))
        ig.sync()
        for q in one:
            want = one[q].cpu().numpy()
            assert np.isfinite(want).all()
            assert rel_err(outs[q].cpu().numpy(), want) <= tol, (k, q)


F1, F2, F3 = [1.4], [1.4, 23.0], [0.408, 1.4, 30.0]
MIXED = {
    "one kind": [("spiral", [4, 8], F2)] * 17,
    "kinds": [("spiral", [2, 8], F2), ("jf12", [2, 8], F2), ("thin", [4], F2),
              ("index", [8], F2)] * 5,
    "pass counts": [("spiral", [4, 8], F1), ("spiral", [8], F2), ("spiral", [8, 4], F3)] * 7,
    "sizes": [("spiral", [1], F2), ("spiral", [64], F2), ("spiral", [16], F2),
              ("jf12", [32, 2], F3)] * 3,
    "one and a group": [("spiral", [8], F1)] * 16 + [("jf12", [8], F1)],
}


@pytest.mark.parametrize("form,tol", [("fp64", 1e-10), ("fp32c", 1e-5)])
@pytest.mark.parametrize("name", list(MIXED))
def test_groups_of_mixed_sets(fields32, form, tol, name):
    rng = np.random.Generator(np.random.PCG64(5))
    ig = _integ(form, fields32)
    entries = _entries(rng, MIXED[name])
    b = ig.batch(entries)
    for _ in range(2):
        b.run()
    ig.sync()
    _check(ig, entries, range(len(entries)), tol)
    b.close()
    ig.close()


@pytest.mark.parametrize("form", ["fp64", "fp32c"])
@pytest.mark.parametrize("nsets,nsides,most", [(200, [8], 13 + 2), (64, [4, 8], 2 * 4 + 3),
                                               (8, [4, 8], 2 + 3)])
def test_kernels_of_a_run(fields32, form, nsets, nsides, most):
    """16 small sets to a kernel, one merge a level and the zeroing."""
    rng = np.random.Generator(np.random.PCG64(6))
    ig = _integ(form, fields32)
    b = ig.batch(_entries(rng, [("spiral", nsides, F2)] * nsets))
    b.run()
    before = ig.launch_count()
    b.run()
    assert ig.launch_count() - before <= most
    b.close()
    ig.close()


@pytest.mark.parametrize("form,nsides,r_max,nsets,shapes", [
    ("fp64", [8], 4.5, 20, 1),      # rays of 45 steps: two lanes whatever is asked for
    ("fp32c", [8], 4.5, 20, 2),     # 1 or 2 lanes, no plan with a grain
    ("fp32c", [8], 4.5, 300, 4),    # the same on the persistent kernel, three grains
])
def test_shapes_that_tuning_times(fields32, form, nsides, r_max, nsets, shapes):
    rng = np.random.Generator(np.random.PCG64(7))
    ig = _integ(form, fields32)
    entries = _entries(rng, [("spiral", nsides, F1)] * nsets)
    for _, o, _ in entries:
        o.radii_shell[1] = r_max * U.kpc
    b = ig.batch(entries, tune=True)
    info = b.info()
    before = ig.launch_count()
    b.run()
    assert info["shapes_tried"] == shapes and info["best_ms"] > 0
    assert info["lanes_per_pixel"] in (1, 2)
    assert (info["grain"] > 0) == (nsets > 256)
    assert ig.launch_count() - before <= (3 if nsets > 256 else 2 + 2)
    _check(ig, entries, [0, nsets - 1], 1e-10 if form == "fp64" else 1e-5)
    b.close()
    ig.close()
