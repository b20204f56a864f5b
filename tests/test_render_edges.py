"""The tiled render where it can go wrong, every kind against the oracle, bit-exact: blocks of 1 (luma is
drawn, the chroma planes have no block and stay as they are), blocks that are not square, planes that end
one sample before and after a tile, motion at the ends of its range."""
import numpy as np
import pytest

from oracle import oracle as orc
from test_render import _cfg

CASES = [  # w, h, block w, block h, step
    (130, 34, 1, 8, 1),
    (130, 34, 8, 1, 2),
    (66, 18, 1, 1, 1),
    (258, 34, 16, 4, 2),
    (254, 30, 4, 32, 1),
    (128, 16, 8, 8, 4),
]


def _inputs(case, seed):
    w, h, bw, bh, step = case
    rng = np.random.default_rng(seed)
    gw, gh = (w - bw // 2) // bw + 1, (h - bh // 2) // bh + 1
    cfg = _cfg(w, h, bw, bh, gw, gh, step)
    n = gw * gh
    ends = np.array([0, 1, 1023, 1024, 1025, 2046, 2047], dtype=np.uint16)
    sets = []
    for _ in range(4):
        pair = []
        for _ in range(2):
            m = rng.integers(1024 - 60, 1024 + 61, size=n).astype(np.uint16)
            at = rng.random(n) < 0.1
            m[at] = rng.choice(ends, size=int(at.sum()))
            pair.append(m)
        sets.append(tuple(pair))
    masks = [rng.integers(0, 256, size=n, dtype=np.uint8) for _ in range(3)]
    planes = []
    for pl in range(3):
        pw, ph = (w // 2, h // 2) if pl else (w, h)
        strides = [pw + 3 * pl, pw + 1]
        planes.append((pw, ph, strides, [rng.integers(0, 256, size=step * step * ph * st, dtype=np.uint8) for st in strides]))
    return cfg, sets, masks, planes, {1: 0, 2: 1, 4: 2}[step]


KINDS = ["warp", "warp mask", "13", "11 mask", "22", "21 final", "23", "23 final"]


def _want(kind, thr, cfg, sets, masks, planes, shift):
    out = []
    for pl, (pw, ph, strides, srcs) in enumerate(planes):
        spans = [st * ph if shift else 0 for st in strides]
        c = pl > 0
        if kind.startswith("warp"):
            out.append(orc.render_warp_plane(cfg, c, True, orc.render_luts(thr)[1], srcs[0], strides[0], spans[0], shift, *sets[0],
                                             pw, ph, masks[0] if "mask" in kind else None))
        elif kind.startswith("23"):
            out.append(orc.render_mode23_plane(cfg, c, True, thr, srcs, strides, spans, shift, sets, masks[:2],
                                               masks[2] if "final" in kind else None, pw, ph))
        else:
            mode = int(kind[:2])
            both = tuple(masks[:2]) if mode > 20 or "mask" in kind else None
            out.append(orc.render_dual_plane(cfg, c, True, False, mode, thr, srcs, strides, spans, shift, sets[0], sets[1], pw, ph,
                                             both, masks[2] if "final" in kind else None, orc.render_threshold_limit(thr, 1.5)))
    return out


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("case", range(3))
def test_oracle_draws_no_chroma_under_blocks_of_one(case, kind):
    want = _want(kind, 200, *_inputs(CASES[case], 900 + case))
    assert want[0].any() and not want[1].any() and not want[2].any()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("case", range(len(CASES)))
def test_render_edges_match_oracle(case, kind):
    import torch

    import svpflow_b200 as sv

    thr = 200 if case % 2 else 256
    inputs = _inputs(CASES[case], 900 + case)
    cfg, sets, masks, planes, shift = inputs
    want = _want(kind, thr, *inputs)
    dev = lambda a: torch.from_numpy(a.astype(np.int16) if a.dtype == np.uint16 else a).cuda()
    src = [[dev(p[3][k]) for p in planes] for k in range(2)]
    one = lambda k: ([t.data_ptr() for t in src[k]], [p[2][k] for p in planes], [t.numel() for t in src[k]])
    dset = [(dev(x), dev(y)) for x, y in sets]
    mot = [(x.data_ptr(), y.data_ptr()) for x, y in dset]
    dm = [dev(m) for m in masks]
    mk = [m.data_ptr() for m in dm]
    dsts = [torch.full((p[1], p[0]), 7, dtype=torch.uint8, device="cuda") for p in planes]
    dp, ds = [d.data_ptr() for d in dsts], [d.shape[1] for d in dsts]
    if kind.startswith("warp"):
        sv.render_warp_device(cfg, thr, False, True, *one(0), shift, *mot[0], dp, ds, mask_ptr=mk[0] if "mask" in kind else 0)
    elif kind.startswith("23"):
        sv.render_mode23_device(cfg, thr, True, *one(0), *one(1), shift, mot, (mk[0], mk[1]), mk[2] if "final" in kind else 0, dp, ds)
    elif int(kind[:2]) > 20:
        sv.render_masked_device(cfg, thr, 1.5, kind[:2] == "22", True, *one(0), *one(1), shift, mot[0], mot[1], (mk[0], mk[1]),
                                mk[2] if "final" in kind else 0, dp, ds)
    else:
        sv.render_blend_device(cfg, thr, kind[:2] == "13", True, False, *one(0), *one(1), shift, mot[0], mot[1], dp, ds,
                               masks=(mk[0], mk[1]) if "mask" in kind else None)
    torch.cuda.synchronize()
    for pl, d in enumerate(dsts):
        drawn = not pl or min(cfg["block_w"], cfg["block_h"]) > 1
        expect = want[pl] if drawn else np.full_like(want[pl], 7)
        got = d.cpu().numpy()
        assert np.array_equal(got, expect), f"plane {pl}: {np.argwhere(got != expect)[:3]}"
