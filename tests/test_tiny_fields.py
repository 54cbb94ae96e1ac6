"""FP64 synchrotron of fields whose squares underflow (a thin disk far from the
plane), CRE index away from 3, where the angle needs 1 / |B_perp|^2.  Against the
CPU oracle for a thin disk (1e-9 of the map maximum, the parity suite's bar), and
against itself for a field scaled by a power of two: with a constant index pe =
(1 + alpha) / 2 and no n_e the maps and the pitch gradient scale by its power pe,
the b0 gradient by pe - 1.  At 2^-465 every square is normal: 1e-9.  At 2^-500 the
squares are subnormal, 5e-324 of at most 1e-313, so the weights of the samples are
good to about 5e-11: 1e-8."""
import numpy as np
import pytest

from conftest import rel_err
from hammurabix_b200 import abi, units as U, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("alpha,beta", [(2.7, 0.0), (2.2, 0.0), (2.7, 0.02)])
def test_thin_disk_vs_oracle(oracle, alpha, beta):
    """B^2 passes through the subnormal range at |z| of 6.9 to 7.2 kpc."""
    from hammurabix_b200.integrator import Integrator
    m = W.spiral_models(hb_kpc=0.02)
    m.cre_ana.alpha, m.cre_ana.beta = alpha, beta
    o = W.make_obs([4, 8], 20.0, 0.05, freq_ghz=23.0)
    ref = oracle.write_grid(o, m)
    with Integrator("fp64") as ig:
        ig.set_models(m)
        got = ig.write_grid(o)
    for k in ("is", "qs", "us"):
        assert np.isfinite(got[k]).all() and got[k].min() > -1e20, k
        assert rel_err(got[k], ref[k]) <= 1e-9, k


def _run(scale, alpha):
    from hammurabix_b200.integrator import Integrator
    m = W.spiral_models()
    m.spiral.b0 *= scale
    m.tereg = abi.HXG_TEREG_NONE
    m.cre_ana.alpha = alpha
    o = W.make_obs([4, 8], 15.0, 0.1, freq_ghz=23.0, do_dm=False, do_fd=False)
    n = abi.npix(8)
    with Integrator("fp64") as ig:
        ig.set_models(m)
        ig.set_checkpointing(True)
        maps = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
        ig.write_grid_device(o, None, None, *maps)
        r = torch.Generator(device="cuda").manual_seed(3)
        g = [torch.rand(n, generator=r, device="cuda", dtype=torch.float64) for _ in range(3)]
        par = torch.zeros(abi.HXG_NUM_PARAMS, dtype=torch.float64, device="cuda")
        ig.adjoint_device(o, None, None, *g, grad_params=par)
        ig.sync()
        return [t.cpu().numpy() for t in maps], par.cpu().numpy()


@pytest.mark.parametrize("alpha", [2.7, 3.0])
@pytest.mark.parametrize("power,tol", [(-465, 1e-9), (-500, 1e-8)])
def test_scaled_field(alpha, power, tol):
    pe = 0.5 * (1.0 + alpha)
    maps, par = _run(1.0, alpha)
    tiny, tpar = _run(2.0 ** power, alpha)
    up = 2.0 ** (-power * pe)
    for a, b in zip(tiny, maps):
        assert np.abs(b).max() > 0
        assert rel_err(a * up, b) <= tol
    for k, f in ((0, up * 2.0 ** power), (1, up), (2, up), (3, up)):
        if abs(par[k]) / f < 1e-290:
            continue                # the scaled gradient is no normal number
        assert abs(tpar[k] * f - par[k]) <= tol * abs(par[k]), k


@pytest.mark.parametrize("alpha", [2.7, 3.0])
@pytest.mark.parametrize("power", [-960, -1000, -1020, -1040])
def test_fields_near_the_smallest_number(alpha, power):
    """Fields of 1e-294 to 1e-318 G: no emission and no gradient, and no NaN."""
    maps, par = _run(2.0 ** power, alpha)
    assert all((t == 0).all() for t in maps)
    assert np.isfinite(par).all()
