"""The transform and demodulator kernels where their layouts change, against
the CPU oracle: windows whose width is no multiple of a tile, of the
demodulator's 8-sample items or of a vector, every carrier phase of the first
sample, rows that start on odd 2-byte boundaries, first lines of either parity
with either field order, windows that touch the field's last sample and line,
per-bin thresholds that differ between a bin and its alias, every output format
behind paddings and buffer offsets that leave rows unaligned, and few enough
lines for the shorter blocks.

Tolerances are those of the full-size cases: chroma within 2e-2 sample units,
floats within 1e-4, integers within one code."""
import numpy as np
import pytest

from oracle import oracle as O
from tests._capture import capture

pytestmark = pytest.mark.gpu

NF = 8
# field width, height, active start, end, first and last frame line, field order
WINDOWS = [
    (301, 61, 40, 301, 4, 119, 0),
    (302, 60, 42, 250, 5, 118, 1),
    (303, 61, 55, 196, 7, 64, 0),
    (304, 40, 37, 46, 2, 75, 1),
    (1135, 40, 185, 1127, 3, 77, 0),
]


def _setup(window, kind, fmt, **kw):
    from libchromadec_gb300 import device as D
    fw, fh, a0, a1, first, last, order = window
    src = capture(NF + 1, 71).fields[order:order + NF]
    x0 = 0 if fw == src.shape[2] else 96      # keeps the burst and a multiple of 4 before the window
    fields = np.ascontiguousarray(src[:, 60:60 + fh, x0:x0 + fw])
    g = D.default_geometry()
    g.field_width, g.field_height, g.active_start, g.active_end = fw, fh, a0, a1
    g.first_active_frame_line, g.last_active_frame_line = first, last
    g.burst_start, g.burst_end = 2, 30
    p = O.params({8: 3, 7: 2, 6: 1}[kind], fmt, first_field_offset=order, **kw)
    for name in ("field_width", "field_height", "active_start", "active_end", "first_active_frame_line",
                 "last_active_frame_line", "burst_start", "burst_end"):
        setattr(p, name, getattr(g, name))
    thr = kw.pop("thresholds", None)
    eng = D.Engine(g, D.default_config(kind=kind, fmt=fmt, thresholds=thr, first_field_offset=order, **kw))
    return eng, p, fields


@pytest.mark.parametrize("kind", [8, 7])
@pytest.mark.parametrize("window", WINDOWS)
def test_chroma(cuda, window, kind):
    torch = cuda
    fw, fh, a0, a1, first, last, order = window
    eng, p, fields = _setup(window, kind, O.FMT_PS)
    n = NF // 2
    lo, hi = first // 2, last // 2 + 1
    out = torch.empty((2 * n, hi - lo, a1 - a0), dtype=torch.float32, device="cuda")
    eng.chroma(torch.from_numpy(fields.reshape(NF, -1).view(np.int16)).cuda(), 0, n, out)
    got = out.cpu().numpy()
    ref = O.transform_chroma(p, fields, 0, n)
    for j in range(2 * n):
        off = (j & 1) ^ order
        b, e = (first + 1 - off) // 2, (last - off) // 2 + 1
        err = np.abs(got[j, b - lo:e - lo] - ref[j, b:e, a0:a1]).max()
        assert err < 2e-2, (j, err)


# kind, format, padding multiple, elements before the frames, luma noise level
DECODES = [(8, O.FMT_P16, 1, 0, 0.0), (7, O.FMT_PS, 8, 1, 0.0), (6, O.FMT_P16, 16, 1, 0.0), (8, O.FMT_RGB48, 8, 2, 0.0),
           (7, O.FMT_RGB48, 1, 3, 0.0), (6, O.FMT_RGBS, 8, 2, 0.0), (7, O.FMT_GRAY16, 4, 1, 0.0),
           (6, O.FMT_GRAYS, 1, 0, 0.0), (8, O.FMT_PS, 2, 0, 1.5), (6, O.FMT_RGB48, 16, 1, 1.5)]


@pytest.mark.parametrize("kind,fmt,padding,shift,nr", DECODES)
@pytest.mark.parametrize("window", WINDOWS)
def test_decode(cuda, window, kind, fmt, padding, shift, nr):
    torch = cuda
    eng, p, fields = _setup(window, kind, fmt, padding_multiple=padding, y_nr_level=nr)
    n = NF // 2
    wide = fmt in (O.FMT_PS, O.FMT_RGBS, O.FMT_GRAYS)
    count = n * eng.frame_bytes // (4 if wide else 2)
    buf = torch.full((count + 16,), 77, dtype=torch.float32 if wide else torch.int16, device="cuda")
    eng.decode(torch.from_numpy(fields.reshape(NF, -1).view(np.int16)).cuda(), 0, n, buf[shift:])
    _check(buf, shift, count, p, fields, wide)


@pytest.mark.parametrize("kind", [8, 7])
@pytest.mark.parametrize("window", WINDOWS)
def test_decode_per_bin(cuda, window, kind):
    """Decoded codes, not chroma: pairs of bins too small to move a sample by
    1/4 unit are left to FP32 decisions, which random thresholds do reach."""
    torch = cuda
    thr = list(np.random.default_rng(3).uniform(0.2, 0.8, 768 if kind == 8 else 80))
    eng, p, fields = _setup(window, kind, O.FMT_P16, thresholds=thr)
    count = (NF // 2) * eng.frame_bytes // 2
    buf = torch.full((count,), 77, dtype=torch.int16, device="cuda")
    eng.decode(torch.from_numpy(fields.reshape(NF, -1).view(np.int16)).cuda(), 0, NF // 2, buf)
    _check(buf, 0, count, p, fields, False)


def _check(buf, shift, count, p, fields, wide):
    host = buf.cpu().numpy()
    assert (host[:shift] == 77).all() and (host[shift + count:] == 77).all()
    ref, _ = O.decode_frames(p, fields, 0, NF // 2, threads=8)
    got = host[shift:shift + count].view(ref.dtype).reshape(ref.shape)
    if wide:
        assert np.abs(got - ref).max() < 1e-4
    else:
        assert np.abs(got.astype(np.int32) - ref.astype(np.int32)).max() <= 1
