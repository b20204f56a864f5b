"""uint16 samples above 1023. The 10-bit extension is defined for 0..1023, but larger samples are not refused: Super and
Analyse give what the oracle's 16-bit build gives for them, wherever they lie (source, reference, a few blocks, all)."""

import numpy as np
import pytest

from oracle import oracle as orc
from payload import first_difference
from test_px16 import clip10

CASES = [  # w, h, super options, analyse options, largest sample, share of 32x32 patches that exceed 1023
    (250, 90, "{pel:4}", "{block:{w:8,overlap:3},main:{search:{type:4,distance:4,satd:true}}}", 4095, 0.2),
    (250, 90, "{pel:2}", "{block:{w:16,overlap:2},main:{search:{type:3,distance:6,satd:true}}}", 4095, 1.0),
    (202, 106, "{pel:2}", "{block:{w:4,overlap:0},main:{search:{type:3,distance:5,satd:true}}}", 65535, 0.3),
    (202, 118, "{pel:2}", "{block:{w:8,overlap:2},refine:[{thsad:100,search:{type:4,distance:2,satd:true}}]}", 16383, 0.1),
    (326, 182, "{pel:1}", "{block:{w:32,overlap:2},main:{search:{type:4,distance:2,satd:false}}}", 1500, 0.3),
    (66, 50, "{pel:2}", "{block:{w:8,overlap:2},main:{search:{type:3,distance:4,satd:true}}}", 2047, 0.5),
]


def _clip(w, h, n, seed, top, share):
    """A 10-bit clip with patches scaled up to `top`, which move from frame to frame."""
    clip = clip10(w, h, n, seed, motion=6, objects=2, object_motion=9).reshape(n, -1)
    rng = np.random.default_rng(seed + 7)
    out = clip.copy()
    for f in range(n):
        off = 0
        for pw, ph in ((w, h), (w // 2, h // 2), (w // 2, h // 2)):
            pl = out[f, off:off + pw * ph].reshape(ph, pw)
            for y in range(0, ph, 32):
                for x in range(0, pw, 32):
                    if rng.random() < share:
                        part = pl[y:y + 32, x:x + 32].astype(np.int64)
                        pl[y:y + 32, x:x + 32] = np.minimum(part * top // 1023 + (part > 900), top)
            off += pw * ph
    assert out.max() > 1023
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("lookahead", [True, False])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_samples_above_1023_match_oracle(case, lookahead):
    import svpflow_b200 as sv

    w, h, sopt, aopt, top, share = CASES[case]
    n = 2
    clip = _clip(w, h, n, 950 + case, top, share)
    sb = sv.Super(w, h, sopt, bits=10)
    an = sv.Analyse(sb.sdata, aopt, w, h, bits=10)
    an.set_lookahead(lookahead)
    so = orc.super_opts(w, h, sopt)
    ao = orc.analyse_opts(orc.sdata(so), aopt, None, w, h)
    supers = orc.build_super_many16(so, clip)
    assert np.array_equal(sb.build_many(clip), supers)
    want = orc.analyse_clip16(ao, so, supers, 0, n)
    got = an.analyse_clip(sb, clip)
    for i in range(n):
        assert got[i].tobytes() == want[i].tobytes(), f"output frame {i}: " + first_difference(got[i], want[i])
