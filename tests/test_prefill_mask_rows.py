"""Prefill attention whose mask rows start on every 2-byte place of a 16-byte piece and end inside a tile, and the rotary
epilogue of a q|k|v projection with fewer strip pairs than SMs, against the one-kernel-per-op plan."""
import numpy as np
import pytest

from conftest import assert_fp16_close
from gehtp_b200.runlists import DecoderConfig, build_decode_runlist, build_prefill_runlist, decode_face
from gehtp_b200.wtop import Engine


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [65, 66, 127, 129, 133, 200, 257, 333])
def test_odd_mask_rows(cuda, tokens):
    cfg = DecoderConfig(256, 1, 4, 2, 128, 512, 256, 1e6, "tiny")
    blob, man = build_prefill_runlist(cfg, tokens, quant="w4")
    ids = (np.arange(tokens) * 7 % cfg.vocab).astype(np.int32)
    out = []
    for fusion in (1, 0):
        cuda.gehtp_cuda_set_fusion(fusion)
        eng = Engine(cuda, blob)
        eng.run_io(ids, man["hidden_temp"])
        out.append(eng.temp(man["hidden_temp"]).reshape(tokens, -1))
        eng.shutdown()
    cuda.gehtp_cuda_set_fusion(1)
    assert_fp16_close(out[0], out[1], "%d tokens" % tokens)
    assert_fp16_close(out[0][-1], out[1][-1], "last of %d tokens" % tokens)      # the row next to the end of the mask


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1, 5])
def test_rotary_epilogue_of_128_strip_pairs(cuda, batch):
    cfg = DecoderConfig(1024, 1, 16, 8, 128, 1024, 256, 1e6, "tiny")              # (16 + 2 * 8) * 128 columns
    blob, man = build_decode_runlist(cfg, batch, 64, quant="w4")
    out = []
    for fusion in (1, 0):
        cuda.gehtp_cuda_set_fusion(fusion)
        cuda.wt_exec_state_reset()
        eng = Engine(cuda, blob)
        for pos in range(3):
            eng.run_io(decode_face(man, np.arange(batch) * 5 + pos, pos, cfg.head_dim, cfg.rope_theta), man["token_temp"])
        out.append(eng.temp(man["logits_temp"]))
        eng.shutdown()
        cuda.wt_exec_state_reset()
    cuda.gehtp_cuda_set_fusion(1)
    assert_fp16_close(out[0], out[1], "batch %d" % batch)
