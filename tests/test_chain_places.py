"""Chains whose result an offset table lays on an input that is dead to the ops by then, but still read by the fused launches: the
two get memory of their own, and results are those of the one-kernel-per-op plan."""
import numpy as np
import pytest

from conftest import assert_fp16_close
from gehtp_b200.runlists import DecoderConfig, Emitter, build_decode_runlist, decode_face
from gehtp_b200.wtop import OP, BlobBuilder, Engine, S


def _apart(cuda, a, b):
    spans = [(cuda.gehtp_cuda_temp_dev(t), cuda.wt_exec_temp_last_bytes(t)) for t in (a, b)]
    (p, m), (q, n) = spans
    return p + m <= q or q + n <= p


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("over", ["k", "v"])
def test_prefill_attention(cuda, hd, over):
    seq, nh, kvh = 200, 4, 2
    rng, e = np.random.default_rng(hd), Emitter()
    src = [e.b.add_slot(rng.standard_normal((seq, n, hd)).astype(np.float16)) for n in (nh, kvh, kvh)]
    mask = np.where(np.tril(np.ones((seq, seq), bool)), 0.0, -np.inf).astype(np.float16)
    mask_b = e.broadcast(S(e.b.add_slot(mask)), (1, 1, seq, seq), (1, nh, seq, seq))
    scale_b = e.broadcast(e.const_f16(hd ** -0.5), (1, 1, 1, 1), (1, 1, 1, nh * seq * seq))
    q, k, v = (e.unary(S(s), seq * n * hd, 14) for s, n in zip(src, (nh, kvh, kvh)))
    qh, kh, vh = e.transpose3(q, (seq, nh, hd), (1, 0, 2)), e.transpose3(k, (seq, kvh, hd), (1, 2, 0)), e.transpose3(v, (seq, kvh, hd), (1, 0, 2))
    s = e.binary(e.bmm(qh, kh, kvh, nh // kvh * seq, hd, seq), scale_b, nh * seq * seq, 2)
    p = e.softmax(e.binary(s, mask_b, nh * seq * seq, 0), nh * seq, seq)
    out = e.transpose3(e.bmm(p, vh, kvh, nh // kvh * seq, seq, hd), (nh, seq, hd), (1, 0, 2))
    n = 2 * seq * nh * hd
    at = {"k": k, "v": v}[over]
    e.b.add_tempoff(4 * n, [(out, 0, n), (at, 0, n // 2), (v if over == "k" else k, n, n // 2)])
    res = []
    for fusion in (1, 0):
        cuda.gehtp_cuda_set_fusion(fusion)
        eng = Engine(cuda, e.b.build())
        eng.run()
        if fusion:
            assert cuda.gehtp_cuda_fused_ops() >= 9 and _apart(cuda, out, at)
        res.append(eng.temp(out))
        eng.shutdown()
    cuda.gehtp_cuda_set_fusion(1)
    assert_fp16_close(res[0], res[1])


@pytest.mark.gpu
def test_rotary_epilogue_of_the_projection(cuda, monkeypatch):
    """Rotated queries on the input of the q|k|v projection whose epilogue writes them."""
    cfg, batch = DecoderConfig(1024, 1, 16, 8, 128, 1024, 256, 1e6, "tiny"), 2
    build = BlobBuilder.build
    ids = {}

    def with_table(b):
        gather = [i for i, (oc, _) in enumerate(b.ops) if oc == OP.KV_APPEND][0]
        lin = [a for oc, a in b.ops[:gather] if oc == OP.MATMUL_W4A16][-1]
        scores = [a for oc, a in b.ops[gather:] if oc == OP.MATMUL_F16][0]
        ids.update(x=lin[0], q=scores[0])
        n = 2 * batch * max(1024, 16 * 128)
        b.add_tempoff(4 * n, [(ids["x"], 0, n), (ids["q"], 0, n)])
        return build(b)
    monkeypatch.setattr(BlobBuilder, "build", with_table)
    blob, man = build_decode_runlist(cfg, batch, 64, quant="w4")
    out = []
    for fusion in (1, 0):
        cuda.gehtp_cuda_set_fusion(fusion)
        cuda.wt_exec_state_reset()
        eng = Engine(cuda, blob)
        for pos in range(3):
            eng.run_io(decode_face(man, np.arange(batch) * 5 + pos, pos, cfg.head_dim, cfg.rope_theta), man["token_temp"])
        if fusion:
            assert _apart(cuda, ids["x"], ids["q"])
        out.append(eng.temp(man["logits_temp"]))
        eng.shutdown()
        cuda.wt_exec_state_reset()
    cuda.gehtp_cuda_set_fusion(1)
    assert_fp16_close(out[0], out[1])
