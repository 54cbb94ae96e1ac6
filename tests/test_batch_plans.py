"""Batches by how their plans are launched: a kernel per parameter set, the
persistent kernel of hundreds of small FP32C sets, and both in one level; the
passes of a set fused or not.  Every entry against the same pass run alone:
1e-10 of the map maximum in FP64 (chunked sums of a few thousand terms), 1e-5 in
FP32C, whose lanes per pixel differ from the single call's."""
import numpy as np
import pytest

from conftest import rel_err
from hammurabix_b200 import abi, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CASES = {
    # name: (Nsides of each parameter set, frequencies, sets checked)
    "one set": ([[8, 16]], [1.4, 23.0], [0]),
    "sets of unequal shells": ([[4], [4, 16], [2, 8, 32], [64]], [0.408, 1.4, 30.0], [0, 1, 2, 3]),
    "single passes": ([[16]] * 3, [1.4], [0, 2]),
    "four passes": ([[8, 16]] * 2, [0.408, 1.4, 5.0, 30.0], [0, 1]),
    "hundreds of small sets": ([[1, 2]] * 300, [1.4, 23.0], [0, 137, 299]),
    "small and large sets": ([[2, 4]] * 280 + [[32, 64]] * 2, [1.4], [0, 200, 280, 281]),
}


@pytest.mark.parametrize("form,tol", [("fp64", 1e-10), ("fp32c", 1e-5)])
@pytest.mark.parametrize("name", list(CASES))
def test_entries_equal_single_passes(fields32, form, tol, name):
    from hammurabix_b200.integrator import Integrator
    shells, freqs, check = CASES[name]
    rng = np.random.Generator(np.random.PCG64(5))
    f64 = [torch.tensor(np.asarray(a, dtype=np.float64).reshape(-1), device="cuda")
           for a in fields32]
    entries, keys = [], ("dm", "fd", "is", "qs", "us")
    for ns in shells:
        m = W.grid_models(W.spiral_models(b0_muG=rng.uniform(2, 8),
                                          pitch_deg=rng.uniform(-40, -5)))
        for o in W.config_grid(ns, 20.0, 0.1, freqs):
            n = abi.obs_output_sizes(o)
            outs = {k: torch.full((c,), np.nan, dtype=torch.float64, device="cuda")
                    for k, c in zip(keys, (n[0], n[1], n[2], n[2], n[2])) if c}
            entries.append((m, o, outs))
    with Integrator(form) as ig:
        ig.set_models(entries[0][0])
        ig.upload_grid_device(abi.HXG_FIELD_BRND, W.grid_desc(32), f64[:3])
        ig.upload_grid_device(abi.HXG_FIELD_TEREG, W.grid_desc(32), f64[3:])
        b = ig.batch(entries)
        for _ in range(2):
            b.run()
        ig.sync()
        for k in check:
            for m, o, outs in entries[k * len(freqs):(k + 1) * len(freqs)]:
                one = {q: torch.zeros_like(t) for q, t in outs.items()}
                ig.set_models(m)
                ig.write_grid_device(o, *(one.get(q) for q in keys))
                ig.sync()
                for q in one:
                    assert rel_err(outs[q].cpu().numpy(), one[q].cpu().numpy()) <= tol, (k, q)
        b.close()
