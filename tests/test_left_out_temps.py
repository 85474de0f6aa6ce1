"""Ops that whole fused runs leave out: whoever reads temps or runs a range behind such a run finds what the one-kernel-per-op
plan leaves, where temp ids are used again, where temps share memory, and in whatever order they are read."""
import ctypes

import numpy as np
import pytest

from gehtp_b200.runlists import DecoderConfig, build_decode_runlist, decode_face
from gehtp_b200.wtop import OP, Engine

CFG = DecoderConfig(512, 1, 8, 4, 64, 512, 2048, 1e6, "small")
B, NSLOTS, RUNS = 3, 77, 4          # a run that plans, one that is captured, two that are replayed
COS, SIN, MASK, COS_Q, MASK_ROWS = 2, 3, 4, 6, 10       # temps of the list below


def _engine(lib):
    buf, man = build_decode_runlist(CFG, B, NSLOTS, seed=3)
    eng = Engine(lib, buf)
    ops = [eng.blob.ops[i] for i in range(eng.blob.n_ops)]
    slices, spread = [i for i, o in enumerate(ops) if o.opcode == OP.SLICE][:4], [i for i, o in enumerate(ops) if o.opcode == OP.BROADCAST]
    assert [ops[i].args[1] for i in slices] == [1, COS, SIN, MASK] and [ops[i].args[1] for i in spread] == [COS_Q, 7, 8, 9, MASK_ROWS, 11]
    return eng, ops, man


def _use_again(ops, old, new):
    """Temp `old` of a slice or broadcast goes by the id of another, whose live range ends before or starts behind it."""
    first = next(i for i, o in enumerate(ops) if o.opcode in (OP.SLICE, OP.BROADCAST) and o.args[1] == old)
    ops[first].args[1] = new
    for o in ops[first + 1:]:
        for k in (0, 1) if o.opcode in (OP.BINARY, OP.ADD) else (0,) if o.opcode == OP.BROADCAST else ():
            if o.args[k] == old:
                o.args[k] = new


def _faces(man):
    rng = np.random.default_rng(5)
    faces = [decode_face(man, rng.integers(0, CFG.vocab, B), p, CFG.head_dim, CFG.rope_theta) for p in range(RUNS)]
    for f in faces:
        f[man["mask_off"]] = np.float16(rng.standard_normal()).view(np.uint16)
    return faces


def _bytes(eng, order):
    got = {}
    for t in order:
        a = eng.temp(t, np.uint8)
        if a is not None:
            got[t] = a
    return got


def _same(got, want, near, skip=0):
    for t in want:
        if t in near:                # sums of the fused chain run in another order: two fp16 roundings of the largest
            a, b = got[t].view(np.float16).astype(np.float32), want[t].view(np.float16).astype(np.float32)
            assert np.abs(a - b).max() <= 2e-2 * np.abs(b).max(), t
        else:
            assert np.array_equal(got[t][skip:], want[t][skip:]), t


def _read_all(lib, reads, change=None):
    """temp -> bytes behind the last of RUNS runs, for each order of `reads`, fused and one kernel per op."""
    out = {}
    for fuse in (1, 0):
        lib.gehtp_cuda_set_fusion(fuse)
        for n, order in enumerate(reads):
            eng, ops, man = _engine(lib)
            eng.state_reset()
            if change:
                change(ops, man)
            for f in _faces(man):
                eng.run_io(f, man["token_temp"], None)
            out[fuse, n] = _bytes(eng, order)
            again = _bytes(eng, order)
            assert all(np.array_equal(again[t], out[fuse, n][t]) for t in again)
            eng.shutdown()
            eng.state_reset()
    lib.gehtp_cuda_set_fusion(1)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("old,new", [(MASK_ROWS, "logits_temp"), (COS_Q, "hidden_temp"), (SIN, "logits_temp"), (MASK_ROWS, 1), (8, 1)])
def test_ids_used_again(cuda, old, new):
    """The id of a broadcast or slice is that of a later result, or of an earlier temp that it takes over."""
    man = _engine(cuda)[2]
    near = {man["logits_temp"], man["hidden_temp"]}
    tid = man.get(new, new)
    temps = sorted({1, COS, SIN, MASK, COS_Q, 7, 8, 9, MASK_ROWS} - {old} | near)
    out = _read_all(cuda, [temps, temps[::-1]], lambda ops, m: _use_again(ops, old, tid))
    for n in (0, 1):
        assert set(out[0, n]) == set(temps)
        _same(out[1, n], out[0, n], near)


@pytest.mark.gpu
@pytest.mark.parametrize("left,over", [(MASK_ROWS, "logits_temp"), (COS_Q, "logits_temp"), (COS, "hidden_temp"), (MASK, "token_temp")])
def test_temps_on_the_same_bytes(cuda, left, over):
    """An offset table lays a broadcast or slice on what a later op writes: all of it, or (tokens) its first bytes."""
    man = _engine(cuda)[2]
    near = {man["logits_temp"], man["hidden_temp"]} | ({left} if over != "token_temp" else set())
    temps = sorted({1, COS, SIN, MASK, COS_Q, 7, 8, 9, MASK_ROWS} | near)
    offs = np.full(4096, 0xFFFFFFFF, np.uint32)
    offs[[left, man[over]]] = 512
    base = np.zeros(16, np.uint8)          # only says that a pool is given
    try:
        out = _read_all(cuda, [temps, temps[::-1]], lambda ops, m: cuda.wt_exec_pool_init(
            base.ctypes.data, 1 << 16, 1 << 15, offs.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32))))
    finally:
        cuda.wt_exec_pool_init(None, 0, 0, None)
    for n in (0, 1):
        _same({t: out[1, n][t] for t in temps}, out[0, n], near, 4 * B if over == "token_temp" else 0)


@pytest.mark.gpu
@pytest.mark.parametrize("first,count,near", [(5, 52, ("logits_temp",)), (9, 48, ("logits_temp",)), (11, 20, (0x17, 0x1e))])
def test_range_behind_a_whole_run(cuda, first, count, near):
    """A range that starts at the broadcasts, among them, or ends inside the attention chain (rotated q and k): it reads what
    the whole run in front of it left out."""
    seen = {}
    for fuse in (1, 0):
        cuda.gehtp_cuda_set_fusion(fuse)
        eng, ops, man = _engine(cuda)
        near = {man.get(t, t) for t in near}
        eng.state_reset()
        for f in _faces(man):
            eng.run_io(f, man["token_temp"], None)
        eng.run_range(first, count)
        seen[fuse] = _bytes(eng, [COS, SIN, MASK, COS_Q, 7, 8, 9, MASK_ROWS, *near])
        eng.shutdown()
        eng.state_reset()
    cuda.gehtp_cuda_set_fusion(1)
    _same(seen[1], seen[0], near)
