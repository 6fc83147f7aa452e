"""Windows that end at the field's last sample on its last line: the tiles there
hang over the end of the field and take its last sample, whatever lies behind
it in memory (the next field, another buffer, nothing). The fields stand
apart with a gap whose contents change; every entry point that transforms them
has to answer the same for both. The chroma is that of the oracle given the
same fields with one more line, all of the last sample (the oracle reads
straight on; the windows hang over by less than a line), within the 2e-2 sample
units of the other windows."""
import numpy as np
import pytest

from oracle import oracle as O
from tests._capture import capture

pytestmark = pytest.mark.gpu

NF = 8
GAP = 64
# field width, height, active start, end, first and last frame line; field order: order 1 puts line fh - 1 in the last field
WINDOWS = [(301, 61, 40, 301, 4, 120, 1), (301, 61, 40, 301, 4, 120, 0), (302, 60, 42, 302, 5, 118, 1),
           (304, 41, 35, 303, 2, 80, 1), (1135, 40, 185, 1127, 3, 78, 1)]


def _setup(window, kind, fmt, thresholds=None):
    from libchromadec_gb300 import device as D
    fw, fh, a0, a1, first, last, order = window
    src = capture(NF + 1, 71).fields[order:order + NF]
    x0 = 0 if fw == src.shape[2] else 96
    fields = np.ascontiguousarray(src[:, 60:60 + fh, x0:x0 + fw])
    g = D.default_geometry()
    g.field_width, g.field_height, g.active_start, g.active_end = fw, fh, a0, a1
    g.first_active_frame_line, g.last_active_frame_line = first, last
    g.burst_start, g.burst_end = 2, 30
    eng = D.Engine(g, D.default_config(kind=kind, fmt=fmt, thresholds=thresholds, first_field_offset=order))
    return eng, g, fields


def _apart(torch, fields, gap_value):
    buf = np.full((NF, fields[0].size + GAP), gap_value, dtype=np.uint16)
    buf[:, :fields[0].size] = fields.reshape(NF, -1)
    return torch.from_numpy(buf.view(np.int16)).cuda()


@pytest.mark.parametrize("kind", [8, 7])
@pytest.mark.parametrize("window", WINDOWS)
def test_chroma(cuda, window, kind):
    torch = cuda
    fw, fh, a0, a1, first, last, order = window
    eng, g, fields = _setup(window, kind, O.FMT_PS)
    n = NF // 2
    lo, hi = first // 2, last // 2 + 1
    got = []
    for gap in (0, 0xFFFF):
        out = torch.empty((2 * n, hi - lo, a1 - a0), dtype=torch.float32, device="cuda")
        eng.chroma(_apart(torch, fields, gap), 0, n, out)
        got.append(out.cpu().numpy())
    p = O.params({8: 3, 7: 2}[kind], O.FMT_PS, first_field_offset=order)
    for name in ("field_width", "active_start", "active_end", "first_active_frame_line", "last_active_frame_line"):
        setattr(p, name, getattr(g, name))
    p.field_height = fh + 1
    taller = np.concatenate([fields, np.broadcast_to(fields[:, -1:, -1:], (NF, 1, fw))], axis=1)
    ref = O.transform_chroma(p, taller, 0, n)
    for j in range(2 * n):
        off = (j & 1) ^ order
        b, e = (first + 1 - off) // 2, (last - off) // 2 + 1
        assert np.array_equal(got[0][j, b - lo:e - lo], got[1][j, b - lo:e - lo]), j
        err = np.abs(got[0][j, b - lo:e - lo] - ref[j, b:e, a0:a1]).max()
        assert err < 2e-2, (j, err)


@pytest.mark.parametrize("kind,per_bin", [(8, False), (8, True), (7, True), (6, False)])
@pytest.mark.parametrize("window", WINDOWS)
def test_decode_takes_nothing_from_behind_a_field(cuda, window, kind, per_bin):
    torch = cuda
    thr = list(np.random.default_rng(3).uniform(0.2, 0.8, 768 if kind == 8 else 80)) if per_bin else None
    eng, g, fields = _setup(window, kind, O.FMT_P16, thr)
    got = []
    for gap in (0, 0xFFFF):
        out = torch.zeros(NF // 2 * eng.frame_bytes // 2, dtype=torch.int16, device="cuda")
        eng.decode(_apart(torch, fields, gap), 0, NF // 2, out)
        got.append(out)
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("window", WINDOWS)
def test_batch_and_features_take_nothing_from_behind_a_field(cuda, window):
    torch = cuda
    from libchromadec_gb300 import device as D
    eng, g, fields = _setup(window, 8, O.FMT_P16)
    order = window[-1]
    batch = D.Batch(g, D.default_config(kind=8, fmt=O.FMT_P16, first_field_offset=order))
    got, feats = [], []
    for gap in (0, 0xFFFF):
        buf = _apart(torch, fields, gap)
        outs = [torch.zeros(NF // 2 * eng.frame_bytes // 2, dtype=torch.int16, device="cuda") for _ in range(2)]
        batch.decode(D.Batch.captures([(buf, 8, 0.4, outs[0]), (buf, 7, 0.5, outs[1])]))
        got.append(torch.stack(outs))
        feat = torch.zeros((NF // 2 + 2, eng.ntiles(), 1280), dtype=torch.int16, device="cuda")
        eng.learned_features(buf, 0, NF // 2, feat)
        feats.append(feat)
    torch.cuda.synchronize()
    assert torch.equal(got[0], got[1])
    assert torch.equal(feats[0], feats[1])
