"""The kernels' dispatch edges against the oracle (integer work: tolerance zero everywhere).

Super's path for packed frames (odd widths, buffers off every alignment, both sample types, the
frame counts and sizes where its launches change), Analyse's walked levels (block shapes and
grids whose levels do not halve evenly, vectors whose reference block leaves the frame, bad-SAD
expansions), the batch's walk (refinement, one direction, more clips than warps of one launch),
the tiled render (planes one sample around its tile), and on the CPU the SATD by a 16 x 16
Sylvester matrix."""
import os

import numpy as np
import pytest

from oracle import oracle as orc
from payload import first_difference
from test_px16 import clip10
from test_render import _gpu_render_case
from test_satd_f16 import satd_int


def _clip(w, h, n, seed, bits=8, **kw):
    from svpflow_b200.synth import make_clip

    return clip10(w, h, n, seed, **kw) if bits > 8 else make_clip(w, h, n, seed=seed, **kw)


@pytest.mark.parametrize("top", [255, 1023])
def test_sylvester_satd_equals_integer_satd(top):
    # samples as halves 1024 + s, products and sums in f32: the bias cancels in H ref - H src, and every
    # partial sum stays below 16 * 2047, which f32 holds exactly
    rng = np.random.default_rng(top)
    src = np.concatenate([rng.integers(0, top + 1, size=(20000, 4, 4)), rng.integers(0, 2, size=(20000, 4, 4)) * top])
    ref = np.concatenate([rng.integers(0, top + 1, size=(20000, 4, 4)), top - src[20000:]])
    h4 = np.array([[1, 1, 1, 1], [1, -1, 1, -1], [1, 1, -1, -1], [1, -1, -1, 1]])
    h16 = np.kron(h4, h4).astype(np.float32)
    half = lambda v: (np.float16(1024) + v.astype(np.float16)).astype(np.float16).astype(np.float32)
    coef = lambda v: half(v).reshape(-1, 16) @ h16
    got = np.abs(coef(ref) - coef(src)).sum(axis=1, dtype=np.float32).astype(np.int64)
    assert np.array_equal(got, satd_int(src, ref))


SUPER_FLAT = [  # w, h, options, bits, frames, buffer offset in samples
    (66, 38, "{pel:2}", 8, 1, 1),
    (98, 54, "{pel:4}", 8, 7, 3),        # one frame more than the cluster tail takes
    (130, 70, "{pel:1}", 8, 6, 5),       # and the most it takes
    (4, 4, "{pel:2}", 8, 2, 0),
    (1026, 62, "{pel:2}", 8, 3, 2),      # a row past a stripe
    (854, 482, "{pel:2, gpu:2}", 8, 2, 7),
    (1282, 722, "{pel:2}", 8, 3, 1),     # large enough for level 0 in a launch of its own
    (66, 38, "{pel:2}", 10, 7, 1),
    (130, 70, "{pel:4}", 10, 1, 3),
    (1282, 722, "{pel:2}", 10, 2, 1),
    (1030, 46, "{pel:1}", 10, 6, 0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(SUPER_FLAT)))
def test_super_packed_matches_oracle(case):
    import torch

    import svpflow_b200 as sv

    w, h, opt, bits, n, off = SUPER_FLAT[case]
    clip = _clip(w, h, n, 700 + case, bits)
    sb = sv.Super(w, h, opt, bits=bits)
    so = orc.super_opts(w, h, opt)
    want = orc.build_super_many16(so, clip) if bits > 8 else orc.build_super_many(so, clip, os.cpu_count() or 1)
    px = 2 if bits > 8 else 1
    src = torch.zeros(clip.nbytes + 64, dtype=torch.uint8, device="cuda")
    dst = torch.full((n * sb.output_len() + 64,), 0x5A, dtype=torch.uint8, device="cuda")
    a, b = off * px, (off + 2) * px
    src[a:a + clip.nbytes] = torch.from_numpy(np.ascontiguousarray(clip).view(np.uint8).reshape(-1)).cuda()
    st = torch.cuda.current_stream().cuda_stream
    sb.build_device(src.data_ptr() + a, dst.data_ptr() + b, n, st)
    out = dst.cpu().numpy()
    got = out[b:b + n * sb.output_len()].copy().view(clip.dtype).reshape(n, -1)
    assert np.array_equal(got, np.asarray(want).reshape(n, -1)), np.argwhere(got != np.asarray(want).reshape(n, -1))[:3]
    assert (out[:b] == 0x5A).all() and (out[b + n * sb.output_len():] == 0x5A).all()  # nothing outside the frames


WALK = [  # w, h, super options, analyse options, frames, bits
    (250, 90, "{pel:2}", "{block:{w:16,h:8,overlap:2},main:{search:{type:3,distance:6,satd:true}}}", 3, 8),
    (118, 214, "{pel:4}", "{block:{w:8,overlap:3},main:{search:{type:4,distance:8,satd:true}}}", 2, 8),
    (202, 106, "{pel:4}", "{block:{w:4,overlap:0},main:{search:{type:3,distance:5,satd:true,coarse:{satd:true}}}}", 2, 8),
    (326, 182, "{pel:2}", "{block:{w:32,overlap:3},main:{search:{type:4,distance:3,satd:true}}}", 2, 8),
    (426, 238, "{pel:1}", "{main:{search:{coarse:{type:4,distance:6,bad:{sad:20,range:-6}}}}}", 2, 8),
    (426, 66, "{pel:2}", "{vectors:2,block:{w:8,overlap:1},main:{search:{coarse:{distance:-8,bad:{sad:30,range:7}}}}}", 9, 8),
    (202, 118, "{pel:2}", "{block:{w:8,overlap:2},refine:[{thsad:100,search:{type:4,distance:2,satd:true}}]}", 2, 8),
    (250, 90, "{pel:4}", "{block:{w:8,overlap:3},main:{search:{type:4,distance:8,satd:true}}}", 2, 10),
    (202, 106, "{pel:2}", "{block:{w:4,overlap:0},main:{search:{type:3,distance:5,satd:true}}}", 2, 10),
    (66, 50, "{pel:2}", "{block:{w:8,overlap:2},main:{search:{type:3,distance:4}}}", 400, 8),  # fewer than 8 warps a direction
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(WALK)))
def test_walk_matches_oracle(case):
    import svpflow_b200 as sv

    w, h, sopt, aopt, n, bits = WALK[case]
    clip = _clip(w, h, n, 800 + case, bits, motion=14, objects=3, object_motion=20)
    sb = sv.Super(w, h, sopt, bits=bits)
    an = sv.Analyse(sb.sdata, aopt, w, h, bits=bits)
    so = orc.super_opts(w, h, sopt)
    ao = orc.analyse_opts(orc.sdata(so), aopt, None, w, h)
    if bits > 8:
        want = orc.analyse_clip16(ao, so, orc.build_super_many16(so, clip), 0, n)
    else:
        want = orc.analyse_clip(ao, so, orc.build_super_many(so, clip, os.cpu_count() or 1), 0, n, os.cpu_count() or 1)
    got = an.analyse_clip(sb, clip)
    for i in range(n):
        assert got[i].tobytes() == want[i].tobytes(), f"output frame {i}: " + first_difference(got[i], want[i])


@pytest.mark.gpu
def test_batch_walk_matches_oracle():
    import svpflow_b200 as sv

    mix = [(202, 118, 4, "{pel:2}", "{block:{w:8,overlap:2},refine:[{thsad:100,search:{type:4,distance:2,satd:true}}]}"),
           (250, 90, 3, "{pel:4}", "{vectors:1,block:{w:16,h:8,overlap:2},main:{search:{type:3,distance:6,satd:true}}}"),
           (66, 50, 600, "{pel:2}", "{vectors:2,block:{w:8,overlap:2},main:{search:{type:3,distance:4}}}"),
           (24, 16, 2, "{pel:1}", "{block:{w:8,overlap:0}}")]  # no level that is walked
    items, clips, want = [], [], []
    for k, (w, h, n, sopt, aopt) in enumerate(mix):
        clip = _clip(w, h, n, 900 + k, motion=6, objects=2, object_motion=9)
        sb = sv.Super(w, h, sopt)
        an = sv.Analyse(sb.sdata, aopt, w, h)
        so = orc.super_opts(w, h, sopt)
        ao = orc.analyse_opts(orc.sdata(so), aopt, None, w, h)
        want.append(orc.analyse_clip(ao, so, orc.build_super_many(so, clip, os.cpu_count() or 1), 0, n, os.cpu_count() or 1))
        items.append((sb, an, n))
        clips.append(clip)
    b = sv.Batch(items)
    try:
        for i, (g, w_) in enumerate(zip(b.run(clips), want)):
            assert np.array_equal(g, w_), f"clip {i} differs from the oracle"
    finally:
        b.close()


RENDER_TILE = [  # as test_render.GPU_CASES: planes of a tile, one sample more and one less, and the chroma planes'
    (128, 16, 8, 1, True, 128, False, 0, False),
    (258, 34, 8, 2, True, 96, True, 3, True),
    (254, 30, 16, 4, True, 200, False, 1, False),
    (130, 18, 4, 2, True, 255, False, 0, True),
    (386, 50, 32, 1, True, 64, True, 5, True),
    (2, 2, 8, 1, True, 128, False, 0, False),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(RENDER_TILE)))
def test_render_tile_matches_oracle(case):
    _gpu_render_case(RENDER_TILE[case], np.random.default_rng(600 + case))
