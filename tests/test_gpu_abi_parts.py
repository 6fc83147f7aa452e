"""Runs of chd_decode_frames_async that are decoded in parts (a quarter, a half
and a quarter, sharing one pinned chunk) deliver the frames that single decodes
give, at run lengths around the one where the parts begin, with a middle part of
any remainder, over the capture's end and past one batch; and a frame stays
whole while its neighbours are freed and the chunk's pool is used again."""
import ctypes

import numpy as np
import pytest

from libchromadec_gb300 import abi, synth
from tests._capture import capture

pytestmark = pytest.mark.gpu

NF = 140


@pytest.fixture(scope="module")
def opened(cuda, tmp_path_factory):
    path = str(tmp_path_factory.mktemp("parts") / "cap.tbc")
    synth.write_tbc(path, capture(NF, 81, dropouts=0.01))
    v = abi.Video(path)
    d = abi.Decoder(v, abi.DEC_TRANSFORM_3D)
    d.set("output_format", "yuv444p16")
    d.commit()
    d.set_dropout(True)
    single = {}

    def frame(k):
        if k not in single:   # a jump decodes one frame
            f = d.decode(k)
            single[k] = f.planes()
            f.close()
        return single[k]

    for k in range(NF // 2 - 1, -1, -1):
        frame(k)
    return d, frame


@pytest.mark.parametrize("first,count", [(0, 9), (3, 10), (60, 10), (5, 11), (1, 14), (0, 23), (3, 64), (2, 65)])
def test_parts_equal_single_frames(opened, first, count):
    d, frame = opened
    got = {i: p for s, i, p in d.decode_async(list(range(first, first + count)))}
    assert sorted(got) == list(range(first, first + count))
    for k in got:
        assert np.array_equal(got[k], frame(k)), k


def test_frames_outlive_the_run(opened):
    d, frame = opened
    held, lib = {}, abi.lib()

    def done(user, status, index, handle):
        assert status == abi.OK
        f = abi.Frame(handle)
        if index in (4, 11, 19):
            held[index] = f
        else:
            f.close()

    cb = abi.FRAME_DONE_CB(done)
    idx = list(range(20))
    arr = (ctypes.c_int64 * 20)(*idx)
    for _ in range(3):   # the chunk of held frames is not reused
        first = dict(held)
        abi.check(lib.chd_decode_frames_async(d._h, arr, 20, cb, None, None), "decode")
        for k, f in first.items():
            assert np.array_equal(f.planes(), frame(k))
            f.close()
    for k, f in held.items():
        assert np.array_equal(f.planes(), frame(k))
        f.close()


def test_cancelled_between_parts(opened):
    d, frame = opened
    for first in (0, 30):   # the second run's uploads follow those the first left behind
        res = d.decode_async(list(range(first, first + 20)), cancel_after=1)
        assert len(res) == 20
        assert res[0][0] == abi.OK and np.array_equal(res[0][2], frame(res[0][1]))
        assert all(s == abi.E_CANCELLED for s, _, _ in res[1:])
    got = {i: p for s, i, p in d.decode_async(list(range(10, 30)))}
    for k in got:
        assert np.array_equal(got[k], frame(k)), k
