"""Decode attention that reads its tables and mask where they lie in the input face: results, and the temps whose ops are
left out, against the one-kernel-per-op plan."""
import numpy as np
import pytest

from gehtp_b200.runlists import DecoderConfig, build_decode_runlist, decode_face
from gehtp_b200.wtop import OP, Engine

CFG = DecoderConfig(512, 2, 8, 4, 64, 512, 2048, 1e6, "small")


@pytest.mark.gpu
@pytest.mark.parametrize("B,nslots", [(1, 64), (3, 77), (8, 130)])
def test_faces_read_in_place(cuda, B, nslots):
    buf, man = build_decode_runlist(CFG, B, nslots, seed=3)
    rng = np.random.default_rng(B)
    faces = [decode_face(man, rng.integers(0, CFG.vocab, B), p, CFG.head_dim, CFG.rope_theta) for p in range(4)]
    for f in faces:
        f[man["mask_off"]:man["mask_off"] + 1] = np.float16(rng.standard_normal()).view(np.uint16)
    logits = np.zeros((B, CFG.vocab), np.float16)
    seen = {}
    for fuse in (0, 1):
        cuda.gehtp_cuda_set_fusion(fuse)
        eng = Engine(cuda, buf)
        eng.state_reset()
        ops = [eng.blob.ops[i] for i in range(eng.blob.n_ops)]
        spread = [o.args[1] for o in ops if o.opcode == OP.BROADCAST][:5]       # cos, sin (q, k) and mask, one row per head
        parts = [o.args[1] for o in ops if o.opcode == OP.SLICE][1:4]           # cos, sin, mask of the face
        got = []
        for i, f in enumerate(faces):
            got.append(eng.run_io(f, man["logits_temp"], logits).copy())
            if i >= 2:          # the graph of the earlier runs did not make these
                got += [eng.temp(t).copy() for t in spread + parts]
        again = np.zeros(B * CFG.n_heads * nslots, np.float16)
        eng.run_io(faces[-1], spread[4], again)
        got.append(again)
        seen[fuse] = got
        eng.shutdown()
        eng.state_reset()
    cuda.gehtp_cuda_set_fusion(1)
    assert len(seen[0]) == len(seen[1])
    for a, b in zip(seen[0], seen[1]):
        if a.shape == logits.shape:      # sums of the fused chain run in another order: two fp16 roundings of the largest
            assert np.abs(a.astype(np.float32) - b.astype(np.float32)).max() <= 2e-2 * np.abs(a.astype(np.float32)).max()
        else:
            assert np.array_equal(a.view(np.uint16), b.view(np.uint16))
