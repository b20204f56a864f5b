"""A server's memory pool: clips of growing size under a tight budget, with the pool's own account of what it holds."""
import ctypes

import numpy as np
import pytest

RESERVED_NOW, RESERVED_HIGH = 5, 6  # CUmemPool_attribute
UNIT = 32 << 20                     # the pool maps device memory in units of 32 MiB


class _Pool:
    def __init__(self):
        import torch

        torch.zeros(1, device="cuda")
        self.cuda = ctypes.CDLL("libcuda.so.1")
        self.h = ctypes.c_void_p()
        assert self.cuda.cuDeviceGetDefaultMemPool(ctypes.byref(self.h), torch.cuda.current_device()) == 0

    def get(self, attr):
        v = ctypes.c_uint64()
        assert self.cuda.cuMemPoolGetAttribute(self.h, attr, ctypes.byref(v)) == 0
        return v.value

    def reset(self):
        assert self.cuda.cuMemPoolTrimTo(self.h, ctypes.c_size_t(0)) == 0
        assert self.cuda.cuMemPoolSetAttribute(self.h, RESERVED_HIGH, ctypes.byref(ctypes.c_uint64(0))) == 0


@pytest.mark.gpu
def test_the_pool_stays_within_the_budget_and_is_given_back():
    import svpflow_b200 as sv
    from svpflow_b200.synth import make_clip

    opt = "{block:{w:8,overlap:3},main:{search:{type:4,distance:24,satd:true}}}"  # searches that outlast the queueing by far
    chunk = 4
    clips = []
    for k, n in enumerate((8, 8, 24)):
        sb = sv.Super(640, 360, "{pel:4}")
        an = sv.Analyse(sb.sdata, opt, 640, 360)
        clips.append((sb, an, make_clip(640, 360, n, seed=40 + k, motion=8, objects=2, object_motion=12)))
    need = [c.nbytes + c.shape[0] * (sb.output_len() + an.payload_len()) + min(4, -(-c.shape[0] // chunk)) * an.scratch_bytes(chunk)
            for sb, an, c in clips]
    budget = int(need[0] + need[1] + 1.3 * need[2])  # all three at once, and less than three of the largest
    pool = _Pool()
    pool.reset()
    before = pool.get(RESERVED_NOW)
    srv = sv.Server(budget, max_active=3, chunk_pairs=chunk)
    try:
        ids = [srv.submit(*c) for c in clips]
        got = [srv.wait(i)[0] for i in ids]
        assert srv.stats()["peak_active"] == 3
        assert pool.get(RESERVED_HIGH) - before <= budget + UNIT
    finally:
        srv.close()
    assert pool.get(RESERVED_NOW) <= before
    for (sb, an, clip), g in zip(clips, got):
        assert np.array_equal(g, an.analyse_clip(sb, clip))
