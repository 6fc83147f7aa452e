"""The input gradients that the training step rounds to bf16, against a chain
of FP32 FMAs in the kernels' stated order: where the tensor cores' sum lies
near a boundary between two bf16 values the step sums again in that order, so
what is rounded is the chain's value. Features, weights and biases are dyadic
fractions, so that every activation is exact in any order; p comes from the
library's own forward pass. From there on each step is restated with its
roundings, and only the weight gradients' FP32 sums over 1,280 voxels a tile
are left: within 1e-5 of the norm (some 40 times 2^-24 times the square root
of 1,280). Energies spread over nine decades, so that single values that fall on
the other side of a boundary move the gradient by more than that: the same
restatement with the sums in the other order shows it. With weights far larger
than the others in a channel without gradient, most values of a tile are near
a boundary, more than the kernel's list holds (2,048)."""
import numpy as np
import pytest

from tests import masknet_ref as R
from tests.test_gpu_masknet import _bf16_bits

pytestmark = pytest.mark.gpu

LIST = 2048
TILES = 6
DARK = 5   # the channel without gradient


def _problem(seed, dark):
    rng = np.random.default_rng(seed)
    P = R.split(R.init_params(seed).astype(np.float64))
    for name, step in (("W1", 2.0 ** -3), ("W2", 2.0 ** -5), ("W3", 2.0 ** -5), ("wh", 2.0 ** -4)):
        P[name] = np.rint(P[name] / step) * step
    P["bh"][:] = 0.25
    if dark:
        P["W2"][:, :, DARK] = 16.0
        P["b2"][DARK] = -65536.0           # a2 of this channel is 0: so is its gradient
        P["W2"][:, DARK, :] = 0.0
        P["W3"][:, :, DARK] = 16.0
        P["W3"][:, DARK, :] = 0.0
        P["b3"][DARK] = -65536.0           # as are a3 and its own
    feat = np.rint(rng.uniform(0.0, 1.0, (TILES, R.NQ, R.NZ, R.NY)) * 8) / 8
    rng = np.random.default_rng(seed + 100)
    a = (np.rint(4.0 * 10.0 ** rng.uniform(0.0, 9.0, feat.shape)) / 4).astype(np.float32).astype(np.float64)   # sums exact in FP64
    c = (a * rng.uniform(-0.2, 1.2, feat.shape)).astype(np.float32)
    return R.join(P).astype(np.float32), feat, a, c


def _chain(d, W, backwards):
    """dA of one tile: d (16, 5, 8, 32), W (27, ci, co); each product and sum rounded once to FP32."""
    acc = np.zeros((R.NC, R.NQ, R.NZ, R.NY), dtype=np.float32)
    order = [(t, co, dq) for t in range(9) for co in range(R.NC) for dq in (-1, 0, 1)]
    for t, co, dq in reversed(order) if backwards else order:
        s = R._shift(d[co], t // 3 - 1, t % 3 - 1, dq)
        w = W[26 - (3 * t + dq + 1), :, co][:, None, None, None]
        acc = (acc.astype(np.float64) + s[None] * w).astype(np.float32)
    return acc


def _near(x, d, W):
    """How many values the kernel's margin calls near a boundary."""
    reach = np.sqrt(sum(R._shift((d * d).sum(0), dz, dy, dq) for _, dz, dy, dq in R._taps()))
    bits = np.ascontiguousarray(x, dtype=np.float32).view(np.uint32)
    dist = np.abs((bits & 0xFFFF).astype(np.int64) - 0x8000) * (bits & 0x7F800000).view(np.float32).astype(np.float64)
    return dist <= 32.0 * np.abs(W).max(axis=(0, 2))[:, None, None, None] * reach[None]


def _gradient(params, feat, a, c, p, backwards=False):
    _, A = R.forward(params.astype(np.float64), feat)
    f32 = np.float32
    inv = f32(1.0 / a.sum())
    dp = f32(2.0) * (p.astype(np.float64) * a - c).astype(f32) * inv   # p a - c: one rounding
    dz = dp * p * (f32(1.0) - p)
    near = []

    def input_gradient(d, W, act):
        out = np.empty(act.shape)
        for t in range(TILES):
            x = _chain(d[t], W, backwards)
            near.append(int((_near(x, d[t], W) & (act[t] > 0)).sum()))
            out[t] = np.where(act[t] > 0, R.bf16(x), 0.0)
        return out

    d3 = np.where(A["a3"] > 0, R.bf16(dz[:, None] * A["wh"].astype(f32)[None, :, None, None, None]), 0.0)
    d2 = input_gradient(d3, A["W3"], A["a2"])
    d1 = input_gradient(d2, A["W2"], A["a1"])
    total = (0, 2, 3, 4)
    g = {"W1": R.conv_w(A["x0"], d1), "b1": d1.sum(total), "W2": R.conv_w(A["a1"], d2), "b2": d2.sum(total),
         "W3": R.conv_w(A["a2"], d3), "b3": d3.sum(total), "wh": np.einsum("bqzy,bcqzy->c", dz.astype(np.float64), A["a3"]),
         "bh": np.array([dz.astype(np.float64).sum()])}
    return g, near


@pytest.mark.parametrize("dark", [False, True])
def test_rounded_as_the_chain(cuda, dark):
    torch = cuda
    from libchromadec_gb300 import device as D
    params, feat, a, c = _problem(23 if dark else 22, dark)   # where the order of summing shows most
    net = D.MaskNet(params)
    f = _bf16_bits(feat.reshape(TILES, -1)).cuda()
    p = torch.empty((TILES, R.NV), dtype=torch.float32, device="cuda")
    net.forward(f, TILES, p)
    net.sync()
    ac = torch.from_numpy(np.stack([a, c], axis=-1).reshape(TILES, R.NV, 2).astype(np.float32)).cuda()
    _, grad = net.train_step(f, ac, TILES, 0.0, want_grad=True)
    net.close()
    pt = p.cpu().numpy().reshape(feat.shape)
    assert np.abs(pt - R.forward(params.astype(np.float64), feat)[0]).max() < 1e-6   # the activations are exact
    want, near = _gradient(params, feat, a, c, pt)
    other, _ = _gradient(params, feat, a, c, pt, backwards=True)
    assert (min(near) > LIST) if dark else (0 < max(near) <= LIST), near
    got = R.split(grad)
    errs = {n: np.linalg.norm(got[n].ravel() - want[n].ravel()) / np.linalg.norm(want[n]) for n, _ in R.SIZES}
    moved = {n: np.linalg.norm(other[n].ravel() - want[n].ravel()) / np.linalg.norm(want[n]) for n, _ in R.SIZES}
    print(errs, moved, near)
    assert max(errs.values()) < 1e-5, errs
    assert max(moved.values()) > 5e-5, moved
