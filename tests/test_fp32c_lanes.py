"""FP32C shells whose rays are cut early and whose launch takes one chunk of the
rays per block, the per-lane sums combined by a second kernel: single and fused
passes, a mask, and the shards of a shell, against the CPU oracle at the FP32C
form's 1e-5 of the map maximum.  At Nside 32 (393216 lanes) the outer shell here
takes that path, the inner one (uncut) does not."""
import numpy as np
import pytest

from conftest import rel_err
from hammurabix_b200 import abi, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KEYS = ("dm", "fd", "is", "qs", "us")


def _passes(freqs, mask):
    passes = W.config_grid([8, 32], 28.0, 0.05, freqs)
    for o in passes:
        o.do_mask = int(mask)
    return passes


def _integ(fields32, m, mask):
    from hammurabix_b200.integrator import Integrator
    ig = Integrator("fp32c")
    ig.set_models(m)
    for slot, (d, comps) in W.grids_dict(32, *fields32).items():
        ig.upload_grid(slot, d, comps)
    if mask is not None:
        ig.set_mask(16, mask)
    return ig


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("freqs", [[23.0], [1.4, 23.0], [1.4, 5.0, 23.0]])
def test_cut_shells_vs_oracle(oracle, fields32, freqs, masked):
    mask = None
    if masked:
        r = np.random.Generator(np.random.PCG64(2))
        mask = (r.random(abi.npix(16)) > 0.4).astype(np.float64)
    m = W.grid_models()
    passes = _passes(freqs, masked)
    ig = _integ(fields32, m, mask)
    got = ig.write_grid_multi(passes)
    ig.close()
    for o, g in zip(passes, got):
        kw = {} if mask is None else dict(mask_nside=16, mask=mask)
        ref = oracle.write_grid(o, m, W.grids_dict(32, *fields32), **kw)
        for k in KEYS:
            if g[k] is not None:
                assert rel_err(g[k], ref[k]) <= 1e-5, k


def test_shards_of_a_cut_shell(fields32):
    """The outer shell's maps of 3 shards (each a launch of its own size) sum to
    the unsplit shell's."""
    m = W.grid_models()
    o = _passes([1.4], False)[0]
    ig = _integ(fields32, m, None)
    n = abi.npix(32)
    z = lambda: [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(5)]  # noqa: E731
    fd = torch.linspace(-1e-2, 1e-2, n, dtype=torch.float64, device="cuda")
    whole, total = z(), z()
    ig.shell_integrate_device(o, 1, 0, 1, fd, whole)
    for s in range(3):
        part = z()
        ig.shell_integrate_device(o, 1, s, 3, fd, part)
        ig.sync()
        for t, p in zip(total, part):
            t += p
    for t, w in zip(total, whole):
        assert w.abs().max() > 0
        assert rel_err(t.cpu().numpy(), w.cpu().numpy()) <= 1e-5
    ig.close()
