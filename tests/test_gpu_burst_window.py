"""Burst windows that leave the line (a capture's metadata sets them): only the
part on the line is read, nothing of the neighbouring lines, fields or memory.
The fields stand in a larger buffer with gaps before, between and behind them
whose contents change; a window that leaves the line on the left gives the
frames of one that starts with the line (the burst there is far above the
detector's floor, the only other thing that the length enters)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests._capture import capture

pytestmark = pytest.mark.gpu

NF, FW, FH, GAP = 4, 301, 61, 192


def _decode(torch, kind, fmt, burst, gap):
    from libchromadec_gb300 import device as D
    fields = capture(NF, 71).fields[:, 60:60 + FH, 96:96 + FW].reshape(NF, -1)
    stride = fields.shape[1] + GAP
    buf = np.full(GAP + NF * stride, gap, dtype=np.uint16)
    buf[GAP:].reshape(NF, stride)[:, :fields.shape[1]] = fields
    dev = torch.from_numpy(buf.view(np.int16)).cuda()
    g = D.default_geometry()
    g.field_width, g.field_height, g.active_start, g.active_end = FW, FH, 40, 290
    g.first_active_frame_line, g.last_active_frame_line = 0, 119
    g.burst_start, g.burst_end = burst
    eng = D.Engine(g, D.default_config(kind=kind, fmt=fmt))
    out = torch.zeros(NF // 2 * eng.frame_bytes, dtype=torch.uint8, device="cuda")
    eng.decode(dev[GAP:].view(NF, stride), 0, NF // 2, out)
    return out


@pytest.mark.parametrize("kind,fmt", [(8, O.FMT_P16), (7, O.FMT_PS), (6, O.FMT_RGB48)])
@pytest.mark.parametrize("burst", [(-10, 30), (280, 320), (-40, 340)])
def test_only_the_line_is_read(cuda, kind, fmt, burst):
    torch = cuda
    a, b = (_decode(torch, kind, fmt, burst, gap) for gap in (0, 0xFFFF))
    assert torch.equal(a, b)
    if burst[1] <= FW:
        assert torch.equal(a, _decode(torch, kind, fmt, (0, burst[1]), 0))
