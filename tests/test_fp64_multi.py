"""FP64 frequency passes in one traversal (hxg_write_grid_multi): every map
against the same pass alone.  A pass's arithmetic is the same in both, so only
the compiler's contraction can differ: a few ulp of a phase of up to 1e4 rad,
1e-11 of the map maximum.  Plus the passes that must stay one by one: with
checkpointing on (the adjoint takes the last pass), and when the shell maps of
all passes do not fit the device."""
import numpy as np
import pytest

from conftest import rel_err
from hammurabix_b200 import abi, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 1e-11


def _maps(o):
    ndm, nfd, nsy = abi.obs_output_sizes(o)
    return [torch.zeros(n, dtype=torch.float64, device="cuda") if n else None
            for n in (ndm, nfd, nsy, nsy, nsy)]


def _integ(fields32, models):
    from hammurabix_b200.integrator import Integrator
    ig = Integrator("fp64")
    ig.set_models(models)
    bx, by, bz, ne = (torch.tensor(np.asarray(a, dtype=np.float64).reshape(-1), device="cuda")
                      for a in fields32)
    if models.brnd == abi.HXG_BRND_GRID:
        ig.upload_grid_device(abi.HXG_FIELD_BRND, W.grid_desc(32), [bx, by, bz])
        ig.upload_grid_device(abi.HXG_FIELD_TEREG, W.grid_desc(32), [ne])
    ig.sync()
    return ig


def _compare(ig, passes):
    fused = [(o, _maps(o)) for o in passes]
    ig.write_grid_multi_device(fused)
    for k, (o, a) in enumerate(fused):
        b = _maps(o)
        ig.write_grid_device(o, *b)
        ig.sync()
        for j in range(5):
            if b[j] is None:
                continue
            x, y = a[j].cpu().numpy(), b[j].cpu().numpy()
            assert np.isfinite(y).all() and (np.abs(y).max() > 0 or j == 1), (k, j)
            assert rel_err(x, y) <= TOL, (k, j, rel_err(x, y))


def _models(kind):
    m = W.spiral_models() if kind in ("analytic", "lsa") else W.grid_models()
    if kind == "lsa":
        m.breg = abi.HXG_BREG_LSA
        m.lsa.b0, m.lsa.psi0, m.lsa.psi1, m.lsa.chi0 = 3e-6, 0.5, 0.02, 0.4
    if kind == "varying index":
        m.cre_ana.beta = 0.02
    if kind == "index 2.6":
        m.cre_ana.alpha = 2.6
    return m


@pytest.mark.parametrize("freqs", [[1.4, 23.0], [0.408, 1.4, 30.0], [0.408, 1.4, 5.0, 30.0]])
@pytest.mark.parametrize("kind", ["analytic", "grid", "lsa", "varying index", "index 2.6"])
def test_fused_passes_equal_single_passes(fields32, kind, freqs):
    ig = _integ(fields32, _models(kind))
    tmpl = W.make_obs([2, 8, 32], 20.0, 0.05, freq_ghz=freqs[-1])
    passes = W.frequency_passes(tmpl, freqs)
    passes[-1].nside_sync = 16          # its own output Nside
    _compare(ig, passes)
    ig.close()


def test_masked_passes(fields32):
    ig = _integ(fields32, _models("grid"))
    rng = np.random.Generator(np.random.PCG64(3))
    ig.set_mask(16, (rng.random(abi.npix(16)) > 0.3).astype(np.float64))
    passes = W.frequency_passes(W.make_obs([8, 16, 32], 20.0, 0.05, freq_ghz=1.4), [1.4, 23.0])
    for o in passes:
        o.do_mask = 1
    _compare(ig, passes)
    ig.close()


def test_checkpointed_passes_stay_single(fields32):
    """With checkpointing on, the adjoint after write_grid_multi differentiates
    the last pass, as after write_grid_device of that pass."""
    passes = W.frequency_passes(W.make_obs([4, 8], 20.0, 0.1, freq_ghz=1.4), [1.4, 23.0])
    got = []
    for multi in (True, False):
        ig = _integ(fields32, _models("grid"))
        ig.set_checkpointing(True)
        outs = [(o, _maps(o)) for o in passes]
        if multi:
            ig.write_grid_multi_device(outs)
        else:
            for o, m in outs:
                ig.write_grid_device(o, *m)
        g = [torch.ones_like(t) if t is not None else None for t in outs[-1][1]]
        par = torch.zeros(abi.HXG_NUM_PARAMS, dtype=torch.float64, device="cuda")
        ig.adjoint_device(passes[-1], *g, grad_params=par)
        ig.sync()
        got.append(par.cpu().numpy())
        ig.close()
    assert np.abs(got[1]).max() > 0
    assert rel_err(got[0], got[1]) <= TOL


def test_passes_that_do_not_fit_together(fields32):
    """Three passes need ten shell maps a shell, one pass four; with room for
    the four only the call runs its passes one by one."""
    ig = _integ(fields32, _models("grid"))
    passes = W.frequency_passes(W.make_obs([256], 2.0, 0.5, freq_ghz=1.4), [0.408, 1.4, 30.0])
    want = []
    for o in passes:
        want.append(_maps(o))
        ig.write_grid_device(o, *want[-1])
    ig.sync()
    outs = [(o, _maps(o)) for o in passes]
    torch.cuda.synchronize()
    hog, room, size = [], 16 << 20, 1 << 33
    while size >= 1 << 21:              # leave less than six maps of 6.3 MB
        if torch.cuda.mem_get_info()[0] - size < room:
            size >>= 1
            continue
        try:
            hog.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            size >>= 1
    ig.write_grid_multi_device(outs)
    ig.sync()
    del hog
    torch.cuda.empty_cache()
    for (o, a), b in zip(outs, want):
        for x, y in zip(a, b):
            if y is not None:
                assert rel_err(x.cpu().numpy(), y.cpu().numpy()) <= TOL
    ig.close()
