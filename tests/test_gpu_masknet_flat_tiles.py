"""Training tiles without energy (black or flat picture: a = c = 0) have no
gradient. They add nothing to a batch's gradient, to the bit, and cost no more
than other tiles: their input gradients are sums of zeros, which no order of
summing rounds differently. An ordinary tile does the same contractions and some
second summing besides, so a batch of flat tiles may take at most twice an
ordinary one's time (the factor is for the clock and the launches)."""
import numpy as np
import pytest

from tests import masknet_ref as R
from tests.test_gpu_masknet import _bf16_bits, _problem

pytestmark = pytest.mark.gpu


def _batch(torch, seed, tiles, flat):
    params, feat, a, c = _problem(seed, tiles)
    ac = np.stack([a, c], axis=-1).reshape(tiles, R.NV, 2).astype(np.float32)
    ac[flat] = 0.0
    return params, _bf16_bits(feat.reshape(tiles, -1)).cuda(), torch.from_numpy(ac).cuda()


@pytest.mark.parametrize("tiles", [2, 40])
def test_flat_tiles_add_nothing(cuda, tiles):
    torch = cuda
    from libchromadec_gb300 import device as D
    params, f, ac = _batch(torch, 9, tiles, slice(1, tiles))
    net = D.MaskNet(params)
    _, alone = net.train_step(f[:1].contiguous(), ac[:1].contiguous(), 1, 0.0, want_grad=True)
    _, grad = net.train_step(f, ac, tiles, 0.0, want_grad=True)
    assert np.array_equal(alone, grad)
    net.close()


@pytest.mark.parametrize("tiles", [32, 304])
def test_flat_tiles_cost_no_more(cuda, tiles):
    torch = cuda
    from libchromadec_gb300 import device as D

    def step_time(ac):
        net.train_step(f, ac, tiles, 0.0, want_loss=False)
        times = []
        for _ in range(9):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            net.train_step(f, ac, tiles, 0.0, want_loss=False)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return float(np.median(times))

    params, f, full = _batch(torch, 9, tiles, slice(0, 0))
    net = D.MaskNet(params)
    flat = full.clone()
    flat[1:] = 0.0
    ordinary = step_time(full)
    assert step_time(flat) < 2.0 * ordinary
    net.close()
