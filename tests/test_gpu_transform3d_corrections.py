"""The corrected outputs of the 3D transform. Three pairs of carriers, one in each
group of columns, stand on bins that mirror onto each other, the second 0.4
times the first: 81 pairs of bins of a tile lie within noise of the threshold,
and FP32 decides some of them wrongly. The counts say that such decisions are
there, in the steps on both sides of the boundary between two chunks of frames
(48) too. The outputs are the oracle's within 1/2 sample unit: a wrong decision
on a carrier's bins moves samples by tens to hundreds, toggling bins that hold
noise only (up to about 30), which the kernels may decide in FP32, by 0.03 a
pair. And they are, to the bit, those of the same frames decoded in launches of
other lengths, where other steps are the first and the last. For a uniform
threshold, a table of them that differ between a bin and its alias and, in a
batch, one for each capture."""
import functools

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

FW, FH, A0, A1, FIRST, LAST = 301, 61, 40, 290, 4, 117
FRAMES, CHUNK = 60, 48


@functools.lru_cache(maxsize=1)
def _fields():
    rng = np.random.default_rng(12)
    x, line = np.arange(FW), np.arange(FH)[:, None]
    f = np.empty((2 * FRAMES, FH, FW), dtype=np.uint16)
    for k in range(2 * FRAMES):
        s = 32000 + 0.5 * rng.standard_normal((FH, FW))
        for kx, ky, kz in ((2, 26, 6), (3, 10, 3), (4, 18, 0)):
            for a, (u, v, w) in ((7000, (kx, ky, kz)), (2800, (8 - kx, 40 - ky, 10 - kz))):
                s = s + a * np.cos(2 * np.pi * (u * x / 16 + v * (2 * line + k % 2) / 32 + w * k / 8))
        f[k] = np.rint(s)
    return f


def _table():
    return list(np.random.default_rng(4).uniform(0.4 - 1e-6, 0.4 + 1e-6, 768))


def _geometry():
    from libchromadec_gb300 import device as D
    g = D.default_geometry()
    g.field_width, g.field_height, g.active_start, g.active_end = FW, FH, A0, A1
    g.first_active_frame_line, g.last_active_frame_line = FIRST, LAST
    g.burst_start, g.burst_end = 2, 30
    return g


def _engine(fmt=O.FMT_PS, **kw):
    from libchromadec_gb300 import device as D
    return D.Engine(_geometry(), D.default_config(kind=8, fmt=fmt, **kw))


def _device(torch):
    return torch.from_numpy(_fields().reshape(2 * FRAMES, -1).view(np.int16)).cuda()


def _decode(torch, eng, fields, first, last):
    out = torch.zeros((last - first) * eng.frame_bytes // 4, dtype=torch.float32, device="cuda")
    eng.decode(fields, first, last, out)
    return out.view(last - first, -1)


@pytest.mark.parametrize("per_bin", [False, True])
def test_corrected_outputs(cuda, per_bin):
    torch = cuda
    kw = {"thresholds": _table()} if per_bin else {"threshold": 0.4}
    fields = _device(torch)
    eng = _engine(**kw)
    lo, hi = FIRST // 2, LAST // 2 + 1
    got = torch.empty((2 * FRAMES, hi - lo, A1 - A0), dtype=torch.float32, device="cuda")
    eng.chroma(fields, 0, FRAMES, got)
    exact, flips = eng.stats()
    print("decisions", exact, "corrected", flips)
    assert flips > FRAMES
    # the frames around the chunks' boundary alone: their own steps and the two before
    for frame in range(CHUNK - 2, CHUNK + 2):
        one = _engine(**kw)
        _decode(torch, one, fields, frame, frame + 1)
        assert one.stats()[1] > 0, frame
    p = O.params(3, O.FMT_PS, **kw)
    for name in ("field_width", "field_height", "active_start", "active_end", "first_active_frame_line",
                 "last_active_frame_line", "burst_start", "burst_end"):
        setattr(p, name, getattr(eng.geometry, name))
    ref = O.transform_chroma(p, _fields(), 0, FRAMES)
    host = got.cpu().numpy()
    for j in range(2 * FRAMES):
        b, e = (FIRST + 1 - (j & 1)) // 2, (LAST - (j & 1)) // 2 + 1
        err = np.abs(host[j, b - lo:e - lo] - ref[j, b:e, A0:A1]).max()
        assert err < 0.5, (j, err)


@pytest.mark.parametrize("per_bin", [False, True])
def test_the_same_in_launches_of_other_lengths(cuda, per_bin):
    torch = cuda
    kw = {"thresholds": _table()} if per_bin else {"threshold": 0.4}
    fields = _device(torch)
    whole = _decode(torch, _engine(**kw), fields, 0, FRAMES)
    for frames in (1, 2, 3, 7, CHUNK):
        eng = _engine(**kw)
        eng.set_max_batch_frames(frames)
        assert torch.equal(_decode(torch, eng, fields, 0, FRAMES), whole), frames
        assert eng.stats()[1] > 0


def test_a_threshold_for_each_capture(cuda):
    torch = cuda
    from libchromadec_gb300 import device as D
    fields = _device(torch)
    batch = D.Batch(_geometry(), D.default_config(kind=8, fmt=O.FMT_PS))
    items, want = [], []
    for thr, first, n in ((0.4, 0, 2 * FRAMES), (0.400001, 4, 40), (0.399999, 10, 2 * FRAMES - 10)):
        own = fields[first:first + n].clone()
        eng = _engine(threshold=thr)
        want.append(_decode(torch, eng, own, 0, n // 2))
        assert eng.stats()[1] > 0, thr
        items.append((own, 8, thr, torch.zeros_like(want[-1])))
    batch.decode(D.Batch.captures(items))
    torch.cuda.synchronize()
    for it, w in zip(items, want):
        assert torch.equal(it[3], w), it[2]
