"""Decode attention over a cached position that is no number: the sequence's logits are none either, those of the others are."""
import numpy as np
import pytest

from conftest import assert_fp16_close
from gehtp_b200.runlists import DecoderConfig, build_decode_runlist, decode_face
from gehtp_b200.wtop import OP, Engine


def _spoil(eng, row, width):
    """The embedding of token `row` becomes NaN throughout."""
    gather = next(op for op in (eng.blob.ops[i] for i in range(eng.blob.n_ops)) if op.opcode == OP.GATHER)
    first = eng.blob.weight_off + eng.blob.slots[gather.args[0] & 0x7FFF].offset + 2 * row * width
    eng.buf[first:first + 2 * width] = np.full(width, np.nan, np.float16).view(np.uint8)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,hd", [(4, 2, 128), (8, 4, 128), (8, 4, 64), (6, 2, 64)])
@pytest.mark.parametrize("slots", [64, 4096])
def test_cached_position_that_is_no_number(cuda, heads, kv_heads, hd, slots):
    cfg, batch, bad = DecoderConfig(256, 1, heads, kv_heads, hd, 512, 256, 1e6, "tiny"), 3, 255
    blob, man = build_decode_runlist(cfg, batch, slots, quant="w4")
    steps = [[3, 9, 27], [4, bad, 28], [5, 11, 29], [6, 12, 30]]
    out = []
    for fusion in (1, 0):
        cuda.gehtp_cuda_set_fusion(fusion)
        cuda.wt_exec_state_reset()
        eng = Engine(cuda, blob)
        _spoil(eng, bad, cfg.hidden)
        for pos, ids in enumerate(steps):
            eng.run_io(decode_face(man, np.array(ids), pos, hd, cfg.rope_theta), man["token_temp"])
        out.append(eng.temp(man["logits_temp"]).reshape(batch, -1))
        eng.shutdown()
        cuda.wt_exec_state_reset()
    cuda.gehtp_cuda_set_fusion(1)
    assert not np.isfinite(out[1][1]).any() and not np.isfinite(out[0][1]).any()
    for b in (0, 2):
        assert_fp16_close(out[0][b], out[1][b], "sequence %d" % b)
