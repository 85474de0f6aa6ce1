"""Decoders with fp16 weights: projections of 16 to 127 rows on the tensor cores and the gated feed-forward in one launch (few
rows) or behind two GEMMs, against the one-kernel-per-op plan; the two products stay readable."""
import numpy as np
import pytest

from conftest import assert_fp16_close
from gehtp_b200.runlists import DecoderConfig, build_decode_runlist, build_prefill_runlist, decode_face
from gehtp_b200.wtop import OP, Engine


def _cfg(hidden, ffn):
    return DecoderConfig(hidden, 1, 4, 2, 128, ffn, 256, 1e6, "tiny")


def _products(eng):
    """The output temps of the gate and the up projection: the two that share input and width."""
    ops = [eng.blob.ops[i] for i in range(eng.blob.n_ops) if eng.blob.ops[i].opcode == OP.MATMUL_F16]
    for a, b in zip(ops, ops[1:]):
        if a.args[0] == b.args[0] and a.args[5] == b.args[5]:
            return [a.args[2], b.args[2]]


@pytest.mark.gpu
@pytest.mark.parametrize("hidden,ffn", [(256, 576), (1024, 4800), (2048, 1088), (512, 19008)])
def test_decode(cuda, hidden, ffn):
    cfg = _cfg(hidden, ffn)
    for batch in (1, 8, 15, 16, 31, 33):
        blob, man = build_decode_runlist(cfg, batch, 64, quant="f16")
        out = []
        for fusion in (1, 0):
            cuda.gehtp_cuda_set_fusion(fusion)
            cuda.wt_exec_state_reset()
            eng = Engine(cuda, blob)
            for pos in range(2):
                eng.run_io(decode_face(man, np.arange(batch) * 5 + pos, pos, cfg.head_dim, cfg.rope_theta), man["token_temp"])
            out.append([eng.temp(man["logits_temp"])] + [eng.temp(t) for t in _products(eng)])
            eng.shutdown()
            cuda.wt_exec_state_reset()
        cuda.gehtp_cuda_set_fusion(1)
        for k, (a, b) in enumerate(zip(*out)):
            assert_fp16_close(a, b, "batch %d, %s" % (batch, ("logits", "gate", "up")[k]))


@pytest.mark.gpu
@pytest.mark.parametrize("hidden,ffn", [(256, 512), (1024, 3072), (2048, 2048)])
@pytest.mark.parametrize("batch", [15, 16, 17, 25, 26, 31, 32])
def test_decode_at_the_line_between_gemv_and_gemm(cuda, hidden, ffn, batch):
    """Widths that both forms take; 1024 x 3072 changes between 25 and 26 rows, 2048 x 2048 between 16 and 17."""
    cfg = _cfg(hidden, ffn)
    blob, man = build_decode_runlist(cfg, batch, 64, quant="f16")
    out = []
    for fusion in (1, 0):
        cuda.gehtp_cuda_set_fusion(fusion)
        cuda.wt_exec_state_reset()
        eng = Engine(cuda, blob)
        for pos in range(2):
            eng.run_io(decode_face(man, np.arange(batch) * 5 + pos, pos, cfg.head_dim, cfg.rope_theta), man["token_temp"])
        out.append([eng.temp(man["logits_temp"])] + [eng.temp(t) for t in _products(eng)])
        eng.shutdown()
        cuda.wt_exec_state_reset()
    cuda.gehtp_cuda_set_fusion(1)
    for k, (a, b) in enumerate(zip(*out)):
        assert_fp16_close(a, b, "batch %d, %s" % (batch, ("logits", "gate", "up")[k]))


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [16, 33, 64, 100, 127, 128])
def test_prefill(cuda, tokens):
    cfg = _cfg(256, 512)
    blob, man = build_prefill_runlist(cfg, tokens, quant="f16")
    ids = (np.arange(tokens) * 7 % cfg.vocab).astype(np.int32)
    out = []
    for fusion in (1, 0):
        cuda.gehtp_cuda_set_fusion(fusion)
        eng = Engine(cuda, blob)
        eng.run_io(ids, man["hidden_temp"])
        out.append(eng.temp(man["logits_temp"]))
        eng.shutdown()
    cuda.gehtp_cuda_set_fusion(1)
    assert_fp16_close(out[0], out[1], "%d tokens" % tokens)
