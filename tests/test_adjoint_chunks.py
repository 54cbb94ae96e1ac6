"""The FP32C adjoint in both of its lane mappings (shells whose rays leave the
cuts early, and late), on pixel counts below and above a block, with a mask and
with the observer off centre, against the FP64 adjoint of the same loss.  Bound:
1e-4 of the largest gradient, the FP32C gradient's own bar (its FP32 samples are
good to a few 1e-6, its sums to 1e-5 at a strong rotation)."""
import numpy as np
import pytest

from conftest import rel_err
from hammurabix_b200 import abi, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _gradient(form, fields32, o, mask):
    from hammurabix_b200.integrator import Integrator
    bx, by, bz, ne = (torch.tensor(np.asarray(a, dtype=np.float64).reshape(-1), device="cuda")
                      for a in fields32)
    m = W.spiral_models()
    m.brnd, m.ternd = abi.HXG_BRND_GRID, abi.HXG_TERND_GRID
    with Integrator(form) as ig:
        ig.set_models(m)
        ig.upload_grid_device(abi.HXG_FIELD_BRND, W.grid_desc(32), [bx, by, bz])
        ig.upload_grid_device(abi.HXG_FIELD_TERND, W.grid_desc(32), [ne - 0.02])
        if mask:
            r = np.random.Generator(np.random.PCG64(4))
            ig.set_mask(8, (r.random(abi.npix(8)) > 0.4).astype(np.float64))
            o.do_mask = 1
        ig.set_checkpointing(True)
        n = abi.obs_output_sizes(o)
        outs = [torch.zeros(c, dtype=torch.float64, device="cuda")
                for c in (n[0], n[1], n[2], n[2], n[2])]
        ig.write_grid_device(o, *outs)
        g = torch.Generator(device="cuda").manual_seed(8)
        up = [torch.randn(t.numel(), generator=g, device="cuda", dtype=torch.float64) / s
              for t, s in zip(outs, (1e21, 1e-1, 1e-2, 1e-2, 1e-2))]
        par = torch.zeros(abi.HXG_NUM_PARAMS, dtype=torch.float64, device="cuda")
        gb = [torch.zeros(32 ** 3, dtype=torch.float64, device="cuda") for _ in range(3)]
        gn = torch.zeros(32 ** 3, dtype=torch.float64, device="cuda")
        ig.adjoint_device(o, *up, grad_params=par, grad_b=gb, grad_ne=gn)
        ig.sync()
        return [t.cpu().numpy() for t in (*gb, gn)], par.cpu().numpy()


@pytest.mark.parametrize("nsides,r_max,observer,mask", [
    ([2], 9.0, W.OBSERVER_KPC, False),        # rays uncut, 48 pixels
    ([2], 30.0, W.OBSERVER_KPC, False),       # cut early
    ([16], 9.0, W.OBSERVER_KPC, True),
    ([16], 30.0, W.OBSERVER_KPC, True),
    ([4, 8, 32], 30.0, (-8.3, 1.0, 4.0), False),
])
def test_fp32c_gradient_in_both_mappings(fields32, nsides, r_max, observer, mask):
    mk = lambda: W.make_obs(nsides, r_max, 0.02, freq_ghz=5.0, observer_kpc=observer)  # noqa: E731
    vox, par = _gradient("fp32c", fields32, mk(), mask)
    vox64, par64 = _gradient("fp64", fields32, mk(), mask)
    for a, b in zip(vox, vox64):
        assert np.abs(b).max() > 0
        assert rel_err(a, b) <= 1e-4
    for k in range(abi.HXG_NUM_PARAMS):
        assert abs(par[k] - par64[k]) <= 1e-4 * abs(par64[k]) + 1e-300, k
