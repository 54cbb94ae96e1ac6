"""FP32C launches that take one chunk of the rays per block and leave per-lane sums to
a second kernel (part_sums: a shell cut early, a launch of at least 896 lanes per SM),
for shards of a shell and with adjoint checkpoints.  A launch on that path counts two
kernels, one below the lane limit a single kernel.  Both take the same 32 chunks a ray
here, so their maps, and the checkpoints behind the gradients, must be the same bits."""
import numpy as np
import pytest

from conftest import rel_err
from hammurabix_b200 import abi, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# a shell from 14 to 28 kpc, 1120 steps, the rays cut from about 10 kpc on
RES, R_MIN, R_MAX = 0.0125, 14.0, 28.0
# Nside, shards on the path (pixels x 32 lanes above 132608), shards off it
SPLITS = [(32, 2, 8), (64, 1, 32), (64, 3, 24), (64, 5, 16)]


def _obs(nside, freq):
    return W.make_obs([nside], R_MAX, RES, freq_ghz=freq, r_min_kpc=R_MIN)


def _integ(fields32, m):
    from hammurabix_b200.integrator import Integrator
    ig = Integrator("fp32c")
    ig.set_models(m)
    bx, by, bz, ne = (torch.tensor(np.asarray(a, dtype=np.float64).reshape(-1), device="cuda")
                      for a in fields32)
    ig.upload_grid_device(abi.HXG_FIELD_BRND, W.grid_desc(32), [bx, by, bz])
    ig.upload_grid_device(abi.HXG_FIELD_TERND if m.ternd else abi.HXG_FIELD_TEREG,
                          W.grid_desc(32), [ne])
    # the grids are packed by the first pass, a launch of its own
    ig.write_grid_device(W.make_obs([1], 1.0, 0.5, do_fd=False), *_zeros(12, 1))
    return ig


def _zeros(n, count):
    return [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(count)]


def _split(ig, nside, shards, kernels, call, maps):
    """The sum over the shards of what call(shard, maps) leaves."""
    total = _zeros(abi.npix(nside), maps)
    for s in range(shards):
        part = _zeros(abi.npix(nside), maps)
        before = ig.launch_count()
        call(s, part)
        assert ig.launch_count() - before == kernels
        ig.sync()
        for t, p in zip(total, part):
            assert int((t * p).count_nonzero()) == 0     # shards share no pixel
            t += p
    return [t.cpu().numpy() for t in total]


@pytest.mark.parametrize("nside,on,off", SPLITS)
@pytest.mark.parametrize("masked", [False, True])
def test_shards_same_bits(fields32, nside, on, off, masked):
    m = W.grid_models()
    ig = _integ(fields32, m)
    o = _obs(nside, 1.4)
    if masked:
        r = np.random.Generator(np.random.PCG64(3))
        ig.set_mask(16, (r.random(abi.npix(16)) > 0.4).astype(np.float64))
        o.do_mask = 1
    fd = torch.linspace(-1e-2, 1e-2, abi.npix(nside), dtype=torch.float64, device="cuda")
    got = [_split(ig, nside, n, k,
                  lambda s, t: ig.shell_integrate_device(o, 0, s, n, fd, t), 5)  # noqa: B023
           for n, k in ((on, 2), (off, 1))]
    for a, b in zip(*got):
        assert np.abs(a).max() > 0 and (a == b).all()
    ig.close()


@pytest.mark.parametrize("nside,on,off", SPLITS)
@pytest.mark.parametrize("freqs", [[1.4, 23.0], [0.408, 1.4, 30.0]])
def test_fused_shards_same_bits(fields32, nside, on, off, freqs):
    ig = _integ(fields32, W.grid_models())
    passes = W.frequency_passes(_obs(nside, 1.4), freqs)
    nf = len(passes)
    fd = torch.linspace(-1e-2, 1e-2, abi.npix(nside), dtype=torch.float64, device="cuda")

    def call(n):
        return lambda s, t: ig.shell_integrate_multi_device(
            passes, 0, s, n, fd, t[0], t[1], [t[2 + 3 * f:5 + 3 * f] for f in range(nf)])
    got = [_split(ig, nside, n, k, call(n), 2 + 3 * nf) for n, k in ((on, 2), (off, 1))]
    for a, b in zip(*got):
        assert np.abs(a).max() > 0 and (a == b).all()
    ig.close()


@pytest.mark.parametrize("nside,on,off", [SPLITS[0], SPLITS[2]])
def test_checkpoints_of_shards(fields32, nside, on, off):
    """Gradients of checkpoints written by the second kernel and by the first: the
    same terms, added by atomics in no fixed order (sums of some 1e5 terms of either
    sign: 1e-10 of the largest)."""
    m = W.spiral_models()
    m.brnd, m.ternd = abi.HXG_BRND_GRID, abi.HXG_TERND_GRID
    o = _obs(nside, 5.0)
    npx, vox = abi.npix(nside), 32 ** 3
    r = torch.Generator(device="cuda").manual_seed(8)
    up = [torch.randn(npx, generator=r, device="cuda", dtype=torch.float64) / s
          for s in (1e21, 1e-1, 1e-2, 1e-2, 1e-2)]
    sums = []
    for n, kernels in ((on, 2), (off, 1)):
        total = np.zeros(abi.HXG_NUM_PARAMS + 4 * vox)
        for s in range(n):
            ig = _integ(fields32, m)
            ig.set_checkpointing(True)
            before = ig.launch_count()
            ig.shell_integrate_device(o, 0, s, n, _zeros(npx, 1)[0], _zeros(npx, 5))
            assert ig.launch_count() - before == kernels
            ig.adjoint_shard_begin(o, s, n)
            ig.adjoint_shard_shell(o, 0, *up, _zeros(npx, 1)[0])
            par, grads = _zeros(abi.HXG_NUM_PARAMS, 1)[0], _zeros(vox, 4)
            ig.adjoint_shard_finish(par, grads[:3], grads[3])
            ig.sync()
            total += torch.cat([par, *grads]).cpu().numpy()
            ig.close()
        sums.append(total)
    a, b = sums
    for k in range(4):
        at = slice(abi.HXG_NUM_PARAMS + k * vox, abi.HXG_NUM_PARAMS + (k + 1) * vox)
        assert np.abs(b[at]).max() > 0 and rel_err(a[at], b[at]) <= 1e-10
    for k in range(abi.HXG_NUM_PARAMS):
        assert abs(a[k] - b[k]) <= 1e-10 * abs(b[k]) + 1e-300, k
