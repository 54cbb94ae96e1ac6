"""Host-buffer calls of one handle: the first small ones through a pageable block,
later ones through pinned memory, larger maps straight into the caller's arrays, in
any order.  Every call's maps are those of the device-buffer call, bit for bit."""
import numpy as np
import pytest

from hammurabix_b200 import abi, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
KEYS = ("dm", "fd", "is", "qs", "us")


@pytest.mark.parametrize("order", [[8] * 20, [2, 64, 4, 8] * 7])
def test_calls_of_one_handle(order):
    from hammurabix_b200.integrator import Integrator
    m = W.spiral_models()
    obs = {n: [W.make_obs([2, n], 20.0, 0.2, freq_ghz=f) for f in (1.4, 23.0)] for n in set(order)}
    want = {}
    with Integrator("fp64") as ig:
        ig.set_models(m)
        for n, passes in obs.items():
            maps = [[torch.zeros(abi.npix(n), dtype=torch.float64, device="cuda")
                     for _ in KEYS] for _ in passes]
            ig.write_grid_multi_device(list(zip(passes, maps)))
            ig.sync()
            want[n] = [[t.cpu().numpy() for t in row] for row in maps]
    with Integrator("fp64") as ig:
        ig.set_models(m)
        for n in order:
            for got, row in zip(ig.write_grid_multi(obs[n]), want[n]):
                for k, t in zip(KEYS, row):
                    assert np.abs(t).max() > 0 and (got[k] == t).all()
