"""Passes of one hxg_write_grid_multi call that write into the same device maps,
as a caller does whose passes all ask for DM and FD and who keeps one of each, or
one set of scratch maps: the result of the passes run in turn, bit for bit where
the passes are one by one and to 1e-11 (FP64) or 1e-5 (FP32C) of the map maximum
where they share a traversal (the fused passes' own bars)."""
import numpy as np
import pytest

from conftest import rel_err
from hammurabix_b200 import abi, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FREQS = [23.0, 5.0, 1.4]


@pytest.mark.parametrize("form,tol", [("fp64", 1e-11), ("fp32c", 1e-5)])
@pytest.mark.parametrize("share", ["fd", "dm and fd", "all", "fd as us"])
@pytest.mark.parametrize("npass", [2, 3])
def test_shared_outputs(fields32, form, tol, share, npass):
    from hammurabix_b200.integrator import Integrator
    passes = [W.make_obs([4, 8, 16], 20.0, 0.1, freq_ghz=f) for f in FREQS[:npass]]
    n = abi.npix(16)
    new = lambda: torch.full((n,), 7.0, dtype=torch.float64, device="cuda")  # noqa: E731

    def maps():
        out = [[new() for _ in range(5)] for _ in passes]
        for m in out[1:]:
            if share in ("fd", "dm and fd", "all"):
                m[1] = out[0][1]
            if share in ("dm and fd", "all"):
                m[0] = out[0][0]
            if share == "all":
                m[2:] = out[0][2:]
            if share == "fd as us":
                m[1] = out[0][4]
        return out
    with Integrator(form) as ig:
        ig.set_models(W.grid_models())
        bx, by, bz, ne = (torch.tensor(np.asarray(a, dtype=np.float64).reshape(-1),
                                       device="cuda") for a in fields32)
        ig.upload_grid_device(abi.HXG_FIELD_BRND, W.grid_desc(32), [bx, by, bz])
        ig.upload_grid_device(abi.HXG_FIELD_TEREG, W.grid_desc(32), [ne])
        got, want = maps(), maps()
        ig.write_grid_multi_device(list(zip(passes, got)))
        for o, m in zip(passes, want):
            ig.write_grid_device(o, *m)
        ig.sync()
    for a, b in zip(got, want):
        for x, y in zip(a, b):
            assert y.abs().max() > 0
            e = rel_err(x.cpu().numpy(), y.cpu().numpy())
            assert e <= (0.0 if share in ("all", "fd as us") else tol), e
