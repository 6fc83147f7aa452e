"""The concealment's luma filter where its sum is an integer, or one unit of the
taps' 1e-8 from one: the integer form and the FP64 form that it falls back to
give the truncation of FIRFilter::apply, byte for byte against the oracle, for
PAL's taps and for those that PAL-M uses, also at the line's ends."""
import numpy as np
import pytest

from libchromadec_gb300 import abi, synth
from oracle import oracle as O
from tests._capture import capture

pytestmark = pytest.mark.gpu

NF = 8
TAPS = {"PAL": (3283437, 23959832, 45513461), "PAL-M": (3275786, 23955702, 45537024)}


def _tuples(c):
    """Five samples whose weighted sum is within 2e-8 of an integer."""
    b = np.arange(0, 131071)
    out = [(0, 0, 0, 0, 0)]
    for a in range(0, 131071, 37):
        k2 = a % 65536
        r = (a * c[0] + b * c[1] + k2 * c[2]) % 10**8
        for v in b[(r <= 2) | (r >= 10**8 - 2)]:
            out.append((a // 2, int(v) // 2, k2, int(v) - int(v) // 2, a - a // 2))
    sums = [(c[0] * (t[0] + t[4]) + c[1] * (t[1] + t[3]) + c[2] * t[2]) % 10**8 for t in out]
    assert sums.count(0) > 4 and len(out) > 20
    return out


@pytest.mark.parametrize("system", ["PAL", "PAL-M"])
def test_sums_at_integers(cuda, tmp_path, system):
    if system == "PAL":
        cap = capture(NF, 91, dropouts=0.05)
    else:
        cap = synth.make_capture(NF, synth.SynthConfig(seed=91, standard="PAL_M", dropout_line_fraction=0.05))
    row = np.array(_tuples(TAPS[system]), dtype=np.uint16).reshape(-1)
    fields = np.empty_like(cap.fields)
    for f in range(NF):
        for y in range(fields.shape[1]):   # a pattern start of its own on every line
            fields[f, y] = np.resize(np.roll(row, 3 * y + f), fields.shape[2])
    cap = synth.SynthCapture(fields=fields, dropouts=cap.dropouts, y=None, u=None, v=None, chroma=None,
                             standard=cap.standard)
    path = str(tmp_path / "cap.tbc")
    synth.write_tbc(path, cap)
    d = abi.Decoder(abi.Video(path), abi.DEC_TRANSFORM_3D)
    d.commit()
    d.set_dropout(True)
    p = O.params(3, O.FMT_P16)
    if system != "PAL":
        p = O.pal_m(p)
    flat = O.flatten_dropouts(cap.dropouts)
    changed = 0
    for k in range(NF // 2):
        ref, _ = O.dropout_correct_frame(p, fields, k, flat)
        assert np.array_equal(d.concealed_fields(k), ref), k
        changed += int((ref != fields[2 * k:2 * k + 2]).sum())
    assert changed > 1000
