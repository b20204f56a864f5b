"""What a user of this framework has it do, as cases that can be timed and compared.

Each case is one kind of call over the sizes and options that the configurations, tests and
benchmark of this repository use it with:

  super    the Super pyramid of a clip's frames that lie on the device
  analyse  the Analyse search over a clip's super frames on the device, one payload per frame
  filter   one output frame of the two filters on host buffers, as a frame server asks for it
  batch    several clips of uneven size analysed in one persistent launch
  smooth   what an interpolator makes of a clip's payloads: scene classes, motion planes, mask
           planes and the rendered frames

Clips are the seeded synthetic ones of svpflow_b200.synth: textured frames with a global motion,
moving rectangles and noise, so that vectors, costs and search lengths are those of real video.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "open-svpflow_b200"))

import svpflow_b200 as sv  # noqa: E402
from svpflow_b200.synth import make_clip_device  # noqa: E402


def listed():
    return [
        # one frame of a small stream: a live source is handed over frame by frame
        {"name": "super_360p_1", "kind": "super", "width": 640, "height": 360, "frames": 1, "pel": 2, "bits": 8},
        # the whole 1080p clip of the benchmark
        {"name": "super_1080p_240", "kind": "super", "width": 1920, "height": 1080, "frames": 240, "pel": 2, "bits": 8},
        # a common web size whose rows are no multiple of 16 bytes, chroma rows of odd length
        {"name": "super_480p_odd_48", "kind": "super", "width": 854, "height": 480, "frames": 48, "pel": 2, "bits": 8},
        # the 10-bit 2160p configuration: uint16 samples, quarter-pel planes
        {"name": "super_2160p10_6", "kind": "super", "width": 3840, "height": 2160, "frames": 6, "pel": 4, "bits": 10},
        # the small 640x360 configuration: 32 frames, hexagon search of radius 2, SAD, full-pel
        {"name": "analyse_360p_32", "kind": "analyse", "width": 640, "height": 360, "frames": 32, "pel": 1, "bits": 8,
         "block": 16, "overlap": 0, "search": 2, "distance": 2, "satd": False, "coarse_satd": False, "refine": 0,
         "vectors": 3},
        # the 1080p configuration, the one the benchmark quotes: UMH of radius 16, SATD + chroma
        {"name": "analyse_1080p_240", "kind": "analyse", "width": 1920, "height": 1080, "frames": 240, "pel": 2,
         "bits": 8, "block": 16, "overlap": 3, "search": 3, "distance": 16, "satd": True, "coarse_satd": True,
         "refine": 0, "vectors": 3},
        # the options of the 10-bit configuration (block 8, exhaustive search of radius 8, quarter-pel)
        # at a frame size whose serial search ends within a second
        {"name": "analyse_360p10_16", "kind": "analyse", "width": 640, "height": 360, "frames": 16, "pel": 4, "bits": 10,
         "block": 8, "overlap": 3, "search": 4, "distance": 8, "satd": True, "coarse_satd": True, "refine": 0,
         "vectors": 3},
        # an odd size with the filter's own defaults and its refinement pass (half-size output blocks)
        {"name": "analyse_480p_refine_48", "kind": "analyse", "width": 854, "height": 480, "frames": 48, "pel": 2,
         "bits": 8, "block": 16, "overlap": 2, "search": 4, "distance": 2, "satd": False, "coarse_satd": True,
         "refine": 200, "vectors": 3},
        # a frame server asks for one 1080p output frame: Super of the new frame, Analyse of the pair
        {"name": "filter_1080p", "kind": "filter", "width": 1920, "height": 1080, "pel": 2, "block": 16, "overlap": 2,
         "vectors": 3},
        # a folder of small clips in one launch, the 1080p search options, blocks of 8 and 16
        {"name": "batch_12_clips", "kind": "batch", "clips": 12, "longest": 40, "largest": 854, "mix": 4},
        # an interpolator's 1080p frames: algorithm 13 (its default) from pel-2 super frames
        {"name": "smooth_1080p_a13_16", "kind": "smooth", "width": 1920, "height": 1080, "frames": 16, "pel": 2,
         "block": 16, "overlap": 3, "algorithm": 13, "masked": False, "phase": 128},
        # the costliest algorithm with all its masks, one frame as it is asked for
        {"name": "smooth_720p_a23_1", "kind": "smooth", "width": 1280, "height": 720, "frames": 1, "pel": 2,
         "block": 16, "overlap": 2, "algorithm": 23, "masked": True, "phase": 96},
    ]


SIZES = [(320, 240), (426, 240), (480, 270), (640, 360), (640, 480), (720, 404), (720, 576), (854, 480), (960, 540),
         (1024, 436), (1280, 546), (1280, 720), (1440, 1080), (1920, 800), (1920, 1080)]


def _log_int(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def _blocks(w, h, block, overlap):
    step = block - (0, block // 8, block // 4, block // 2)[overlap]
    return (w // step) * (h // step)


def draw(rng):
    kind = rng.choice(["super", "super", "analyse", "analyse", "analyse", "filter", "batch", "smooth", "smooth"])
    w, h = rng.choice(SIZES)
    if rng.random() < 0.4:  # a cropped picture: any even size
        w -= 2 * rng.randrange(1, 40)
        h -= 2 * rng.randrange(1, 30)
    if kind == "super":
        bits = rng.choice([8, 8, 8, 10])
        pel = rng.choice([1, 2, 2, 4])
        most = max(1, int(2.5e9 / (w * h * pel * pel * 1.5 * (2 if bits == 10 else 1))))
        return {"kind": kind, "width": w, "height": h, "frames": _log_int(rng, 1, min(240, most)), "pel": pel,
                "bits": bits}
    if kind == "analyse":
        bits = rng.choice([8, 8, 8, 10])
        pel = rng.choice([1, 2, 2, 4])
        block, overlap = rng.choice([8, 16, 16, 32]), rng.choice([0, 1, 2, 2, 3])
        search = rng.choice([2, 3, 3, 4])
        distance = {2: rng.choice([2, 4, 8]), 3: rng.choice([4, 8, 12, 16]), 4: rng.choice([2, 3, 4, 8])}[search]
        satd, refine = rng.random() < 0.6, 0
        if block >= 16 and rng.random() < 0.25:
            refine = rng.choice([200, 400])
        tall = 33000 / (1 if bits == 8 else 3) / (4 if refine else 1) / (2 if distance == 8 and search == 4 else 1)
        while _blocks(w, h, block, overlap) > tall:  # the search is a chain over the blocks
            w, h = max(160, w // 4 * 2), max(120, h // 4 * 2)
            if w == 160 and h == 120:
                break
        most = max(1, min(240, int(7.7e6 / _blocks(w, h, block, overlap) / (1 if bits == 8 else 3) / (4 if refine else 1))))
        return {"kind": kind, "width": w, "height": h, "frames": _log_int(rng, 1, most), "pel": pel, "bits": bits,
                "block": block, "overlap": overlap, "search": search, "distance": distance, "satd": satd,
                "coarse_satd": rng.random() < 0.7, "refine": refine, "vectors": rng.choice([1, 2, 3, 3])}
    if kind == "filter":
        return {"kind": kind, "width": w, "height": h, "pel": rng.choice([1, 2, 2, 4]), "block": rng.choice([16, 16, 32]),
                "overlap": rng.choice([0, 1, 2]), "vectors": rng.choice([1, 2, 3, 3])}
    if kind == "batch":
        return {"kind": kind, "clips": rng.randrange(2, 17), "longest": _log_int(rng, 8, 60),
                "largest": rng.choice([480, 640, 854]), "mix": rng.randrange(1 << 20)}
    return {"kind": kind, "width": w, "height": h, "frames": _log_int(rng, 1, 16), "pel": rng.choice([1, 2, 2, 4]),
            "block": rng.choice([8, 16, 16, 32]), "overlap": rng.choice([0, 2, 3]),
            "algorithm": rng.choice([1, 2, 11, 13, 13, 21, 22, 23]), "masked": rng.random() < 0.5,
            "phase": rng.randrange(1, 256)}


class _View:
    """A buffer that an object of the framework owns on the device, as torch.as_tensor takes it. The
    tensor keeps the view alive, and the view the owner."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (ptr, False), "version": 3}


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _clip(case, frames, seed):
    bits = case.get("bits", 8)
    return make_clip_device(case["width"], case["height"], frames, seed, motion=24, objects=8, object_motion=48,
                            noise=2.0 if bits == 8 else 8.0, bits=bits)


def _bool(v):
    return "true" if v else "false"


def _analyse_opt(case):
    refine = ",refine:[{thsad:%d}]" % case["refine"] if case["refine"] else ""
    return "{block:{w:%d,overlap:%d},vectors:%d,main:{search:{type:%d,distance:%d,satd:%s,coarse:{satd:%s}}}%s}" % (
        case["block"], case["overlap"], case["vectors"], case["search"], case["distance"], _bool(case["satd"]),
        _bool(case["coarse_satd"]), refine)


def _mix(case):
    """The batch's clips: (width, height, frames, block, seed offset)."""
    rng = random.Random(case["mix"])
    sizes = [s for s in ((320, 240), (426, 240), (480, 270), (640, 360), (854, 480)) if s[0] <= case["largest"]]
    clips = []
    for i in range(case["clips"]):
        w, h = rng.choice(sizes)
        block = 16 if w > 480 else rng.choice([8, 16])
        clips.append((w, h, _log_int(rng, 4, case["longest"]), block, i))
    return clips


def _super_on_device(sb, frames):
    n = frames.shape[0]
    supers = torch.zeros(n, sb.output_len(), dtype=torch.uint8, device="cuda")
    sb.build_device(frames.data_ptr(), supers.data_ptr(), n, _stream())
    return supers


def prepare(case, seed):
    kind = case["kind"]
    if kind == "super":
        sb = sv.Super(case["width"], case["height"], "{pel:%d}" % case["pel"], bits=case["bits"])
        frames = _clip(case, case["frames"], seed)
        return {"kind": kind, "sb": sb, "frames": frames,
                "supers": torch.zeros(case["frames"], sb.output_len(), dtype=torch.uint8, device="cuda")}
    if kind == "analyse":
        sb = sv.Super(case["width"], case["height"], "{pel:%d}" % case["pel"], bits=case["bits"])
        an = sv.Analyse(sb.sdata, _analyse_opt(case), case["width"], case["height"], bits=case["bits"])
        n = case["frames"]
        supers = _super_on_device(sb, _clip(case, n, seed))
        return {"kind": kind, "an": an, "supers": supers, "frames": n,
                "payloads": torch.zeros(n, an.payload_len(), dtype=torch.uint8, device="cuda"),
                "scratch": torch.zeros(an.scratch_bytes(n), dtype=torch.uint8, device="cuda")}
    if kind == "filter":
        sb = sv.SuperBuilder(case["width"], case["height"], case["pel"])
        an = sv.Analyser(sb, case["block"], case["block"], case["overlap"], case["vectors"])
        frames = _clip(case, 2, seed).cpu().numpy()
        return {"kind": kind, "sb": sb, "an": an, "last": sb.build(frames[0]), "next": frames[1]}
    if kind == "batch":
        clips, mix = [], _mix(case)
        for w, h, n, block, _ in mix:
            sb = sv.Super(w, h, "{pel:2}")
            opt = "{block:{w:%d,overlap:3},main:{search:{type:3,distance:16,satd:true}}}" % block
            clips.append((sb, sv.Analyse(sb.sdata, opt, w, h), n))
        b = sv.Batch(clips)
        for i, (w, h, n, block, k) in enumerate(mix):
            frames = _clip({"width": w, "height": h}, n, seed * 64 + k)
            torch.as_tensor(_View(b, b.frames_device(i), frames.numel()), device="cuda").copy_(frames.reshape(-1))
        torch.cuda.synchronize()
        return {"kind": kind, "batch": b, "payloads": [
            torch.as_tensor(_View(b, b.payloads_device(i), c[2] * c[1].payload_len()), device="cuda")
            for i, c in enumerate(clips)]}
    w, h, n = case["width"], case["height"], case["frames"]
    sb = sv.Super(w, h, "{pel:%d}" % case["pel"])
    an = sv.Analyse(sb.sdata, "{block:{w:%d,overlap:%d},main:{search:{type:2,distance:2}}}" % (
        case["block"], case["overlap"]), w, h)
    # algorithm 23 reads the payloads on both sides of a frame's own
    supers = _super_on_device(sb, _clip(case, n + 3, seed))
    payloads = torch.zeros(n + 2, an.payload_len(), dtype=torch.uint8, device="cuda")
    scratch = torch.zeros(an.scratch_bytes(n + 2), dtype=torch.uint8, device="cuda")
    an.analyse_clip_device(supers.data_ptr(), n + 3, 0, n + 2, payloads.data_ptr(), scratch.data_ptr(), _stream())
    an.device_status(scratch.data_ptr(), _stream())
    vd = an.vector_header()
    gw, gh = sv.vector_grid(vd)
    hs = sb.super_height
    return {"kind": kind, "case": dict(case), "vd": vd, "n": n, "grid": gw * gh, "supers": supers, "payloads": payloads,
            "cfg": dict(width=w, height=h, block_w=vd[2] - vd[9], block_h=vd[3] - vd[10], origin_x=vd[2] // 2,
                        origin_y=vd[3] // 2, grid_w=gw, grid_h=gh, source_step=case["pel"]),
            "shift": {1: 0, 2: 1, 4: 2}[case["pel"]], "strides": [w, w // 2, w // 2],
            "offs": [0, w * hs, w * hs + (w // 2) * (hs // 2)],
            "lens": [w * hs, (w // 2) * (hs // 2), (w // 2) * (hs // 2)],
            "out_offs": [0, w * h, w * h + (w // 2) * (h // 2)],
            "planes": torch.zeros(n + 2, 4 * gw * gh, dtype=torch.int16, device="cuda"),
            "masks": torch.zeros(n + 2, 5 * gw * gh, dtype=torch.uint8, device="cuda"),
            "mask_scratch": torch.zeros(sv.render_masks_scratch(vd, n + 2), dtype=torch.uint8, device="cuda"),
            "classes": torch.zeros(n + 2, dtype=torch.int32, device="cuda"),
            "status": torch.zeros(3, n + 2, dtype=torch.int32, device="cuda"),
            "out": torch.zeros(n, w * h + 2 * (w // 2) * (h // 2), dtype=torch.uint8, device="cuda")}


def _smooth(s):
    case, vd, m, st = s["case"], s["vd"], s["grid"], _stream()
    thr, algorithm, scale = case["phase"], case["algorithm"], 0.01
    pay, np_, plen = s["payloads"].data_ptr(), s["n"] + 2, s["payloads"].shape[1]
    status = [s["status"][i].data_ptr() for i in range(3)]
    sv.scene_class_device(vd, pay, plen, np_, s["classes"].data_ptr(), status[0], stream=st)
    sv.vector_planes_device(vd, pay, plen, np_, case["width"], case["height"], s["planes"].data_ptr(), status[1], stream=st)
    masked = case["masked"] or algorithm >= 21
    if masked:
        sv.render_masks_device(vd, pay, plen, np_, thr, s["masks"].data_ptr(), s["mask_scratch"].data_ptr(), status[2],
                               cover=100, area_scale=scale, stream=st)
    sup, plane, mask, out = (s[k].data_ptr() for k in ("supers", "planes", "masks", "out"))
    sup_len, plane_len, mask_len, out_len = s["supers"].shape[1], 8 * m, 5 * m, s["out"].shape[1]
    cfg, lens, strides, shift = s["cfg"], s["lens"], s["strides"], s["shift"]
    for i in range(s["n"]):
        f = i + 1  # payload f lies between frames f and f + 1
        src0 = [sup + f * sup_len + o for o in s["offs"]]
        src1 = [sup + (f + 1) * sup_len + o for o in s["offs"]]
        dst = [out + i * out_len + o for o in s["out_offs"]]
        # a payload's planes: x and y of the previous set, then of the current one
        sets = lambda k, cur: (plane + k * plane_len + cur * 4 * m, plane + k * plane_len + cur * 4 * m + 2 * m)  # noqa: E731
        mk = mask + f * mask_len  # cover0, cover1, area0, area1, area_max
        if algorithm in (1, 2):
            one = algorithm == 1
            sv.render_warp_device(cfg, thr, one, True, src1 if one else src0, strides, lens, shift, *sets(f, int(one)),
                                  dst, strides, st, (mk + (2 if one else 3) * m) if masked else 0)
        elif algorithm in (11, 13):
            sv.render_blend_device(cfg, thr, algorithm == 13, True, False, src0, strides, lens, src1, strides, lens,
                                   shift, sets(f, 0), sets(f, 1), dst, strides,
                                   (mk + 2 * m, mk + 3 * m) if masked else None, st)
        elif algorithm in (21, 22):
            sv.render_masked_device(cfg, thr, scale, algorithm == 22, True, src0, strides, lens, src1, strides, lens,
                                    shift, sets(f, 0), sets(f, 1), (mk, mk + m), mk + 4 * m if case["masked"] else 0,
                                    dst, strides, st)
        else:
            sv.render_mode23_device(cfg, thr, True, src0, strides, lens, src1, strides, lens, shift,
                                    (sets(f, 0), sets(f, 1), sets(f + 1, 0), sets(f - 1, 1)), (mk, mk + m),
                                    mk + 4 * m if case["masked"] else 0, dst, strides, st)
    got = {"frames": s["out"], "planes": s["planes"], "classes": s["classes"], "status": s["status"]}
    if masked:
        got["masks"] = s["masks"]
    return got


def run(state):
    kind = state["kind"]
    if kind == "super":
        state["sb"].build_device(state["frames"].data_ptr(), state["supers"].data_ptr(), state["frames"].shape[0], _stream())
        return state["supers"]
    if kind == "analyse":
        n = state["frames"]
        state["an"].analyse_clip_device(state["supers"].data_ptr(), n, 0, n, state["payloads"].data_ptr(),
                                        state["scratch"].data_ptr(), _stream())
        return state["payloads"]
    if kind == "filter":
        cur = state["sb"].build(state["next"])
        payload = state["an"].analyse(state["last"], cur)
        return {"super": cur.data, "payload": np.frombuffer(payload, dtype=np.uint8)}
    if kind == "batch":
        state["batch"].launch()
        state["batch"].status()  # the launch runs on the batch's own stream: waits for it and reports
        return state["payloads"]
    return _smooth(state)


def _search_flops(w, h, block, overlap, search, distance, satd):
    """Operations of one direction's search of one pair: 2 per SAD sample, 111 per SATD 4x4 tile, luma and
    chroma, over the candidates of every block (special ones, the pattern, hexagon and ring steps) and a third
    more for the coarser levels."""
    tried = 8 + {2: 20, 3: 4 * (distance // 2) + 16 * max(distance // 4, 1) + 14, 4: (2 * distance + 1) ** 2}[search]
    per_sample = 111 / 16 if satd else 2
    return _blocks(w, h, block, overlap) * tried * block * block * 1.5 * per_sample * 4 / 3


def _super_bytes(w, h, pel, sample):
    """A super frame: the pel planes of level 0 and a third of a plane for the levels above it."""
    return w * h * 1.5 * (pel * pel + 1 / 3) * sample


def work(case):
    kind = case["kind"]
    if kind == "super":
        w, h, sample = case["width"], case["height"], 2 if case["bits"] == 10 else 1
        return {"bytes": case["frames"] * (w * h * 1.5 * sample + _super_bytes(w, h, case["pel"], sample)), "flops": 0}
    if kind == "analyse":
        w, h, n, sample = case["width"], case["height"], case["frames"], 2 if case["bits"] == 10 else 1
        dirs = 2 if case["vectors"] == 3 else 1
        payload = dirs * 8 * _blocks(w, h, case["block"], case["overlap"]) * (4 if case["refine"] else 1)
        flops = _search_flops(w, h, case["block"], case["overlap"], case["search"], case["distance"], case["satd"])
        return {"bytes": n * (_super_bytes(w, h, case["pel"], sample) + payload), "flops": n * dirs * flops}
    if kind == "filter":
        w, h = case["width"], case["height"]
        dirs = 2 if case["vectors"] == 3 else 1
        payload = dirs * 8 * _blocks(w, h, case["block"], case["overlap"])
        return {"bytes": w * h * 1.5 + 3 * _super_bytes(w, h, case["pel"], 1) + payload,
                "flops": dirs * _search_flops(w, h, case["block"], case["overlap"], 4, 2, False)}
    if kind == "batch":
        total = {"bytes": 0, "flops": 0}
        for w, h, n, block, _ in _mix(case):
            total["bytes"] += n * (w * h * 1.5 + 2 * _super_bytes(w, h, 2, 1) + 16 * _blocks(w, h, block, 3))
            total["flops"] += n * 2 * _search_flops(w, h, block, 3, 3, 16, True)
        return total
    w, h, n = case["width"], case["height"], case["frames"]
    reads = 1 if case["algorithm"] in (1, 2) else 2  # source frames that a rendered one samples
    grid = _blocks(w, h, case["block"], case["overlap"])
    return {"bytes": n * w * h * 1.5 * (reads + 1) + (n + 2) * grid * (16 + 8 + 5), "flops": n * w * h * 1.5 * 20 * reads}


def exact(case, seed):
    """Every output is a byte or a whole number (samples, vectors, scores, classes): there is no value in 64
    bits that it comes near to, it is equal or wrong."""
    return None
