"""The tensor-core backward pass over more tiles than thread blocks run at
once: a batch that repeats five tiles has the loss and the gradient of the
five (the loss is normalised by the batch's energy), for one tile a block,
for several, and for a count that leaves some blocks one fewer. Against the
FP64 restatement with its rounding points, at the tolerance of the five-tile
test (the forward pass's own bf16 activations)."""
import numpy as np
import pytest

from tests import masknet_ref as R
from tests.test_gpu_masknet import _bf16_bits, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("repeats", [1, 2, 61, 130])
def test_gradient_of_repeated_tiles(cuda, repeats):
    torch = cuda
    from libchromadec_gb300 import device as D
    params, feat, a, c = _problem(9, 5)
    net = D.MaskNet(params)
    f = _bf16_bits(feat.reshape(5, -1)).cuda().repeat(repeats, 1)
    ac = torch.from_numpy(np.stack([a, c], axis=-1).reshape(5, R.NV, 2).astype(np.float32)).cuda().repeat(repeats, 1, 1)
    loss, grad = net.train_step(f, ac, 5 * repeats, 0.0, want_grad=True)
    L, gref, _ = R.loss_and_grad(params.astype(np.float64), feat, a, c)
    assert abs(loss - L) <= 1e-4 * abs(L), (loss, L)
    o = 0
    for name, n in R.SIZES:
        g, r = grad[o:o + n].astype(np.float64), gref[o:o + n]
        assert np.linalg.norm(g - r) < 1e-2 * np.linalg.norm(r), name
        o += n
    net.close()
