"""The learned form's network on the repeating half of each tile: the engine's
decode (which runs the network on ky < 16 of two tiles at a time) equals the
passes run by hand with the network over whole tiles, bit for bit -- also when
the tile count is odd and the last pair has one tile, and at either parity of
the first field's rows."""
import os

import numpy as np
import pytest

from tests._capture import capture

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,first_line,frames", [(948, 44, 2), (940, 44, 1), (941, 45, 1), (24, 44, 3)])
def test_half_network_equals_whole(cuda, width, first_line, frames):
    torch = cuda
    from libchromadec_gb300 import device as D
    src = capture(12, 33)
    f = torch.from_numpy(src.fields.reshape(12, -1).view(np.int16)).cuda()
    g = D.default_geometry()
    g.active_end = g.active_start + width
    g.first_active_frame_line = first_line
    w = np.fromfile(os.path.join(os.path.dirname(D.__file__), "data", "tpal3d_masknet.f32"), dtype="<f4")
    net = D.MaskNet(w)
    eng = D.Engine(g, D.default_config(kind=D.KIND_TRANSFORM_3D, fmt=D.FMT_PS))
    nt = eng.ntiles() * (frames + 2)
    feat = torch.empty((nt, D.MASKNET_BINS), dtype=torch.int16, device="cuda")
    p = torch.empty((nt, D.MASKNET_BINS), dtype=torch.float32, device="cuda")
    fb = torch.empty(nt, dtype=torch.uint8, device="cuda")
    rows = g.last_active_frame_line // 2 + 1 - first_line // 2
    whole = torch.empty((2 * frames, rows, width), dtype=torch.float32, device="cuda")
    half = torch.empty_like(whole)
    eng.learned_features(f, 2, 2 + frames, feat)
    net.forward(feat, nt, p, fb)
    eng.learned_chroma(f, 2, 2 + frames, p, fb, whole)
    q = p.view(nt, 5, 8, 32)
    assert torch.equal(q, q.roll((4, 16), (2, 3)))     # the repeat itself
    eng.set_masknet(net)
    eng.chroma(f, 2, 2 + frames, half)
    net.sync()
    assert torch.equal(half, whole)
    tiles, fallback = eng.learned_stats()
    assert tiles == nt and fallback == int(fb.sum())
