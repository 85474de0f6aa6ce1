"""Values that are not finite: a row's result holds nothing of tokens behind it, and infinite scores and weights count as in
plain fp32 arithmetic, however kernels cut rows, keys and sums."""
import numpy as np
import pytest

import ripidra_oracle
import supevik_oracle
import test_ripidra as rip
import test_supevik as sup
from gehtp_b200.checkpoint import bf16_to_f32, f32_to_bf16
from gehtp_b200.rowlists import RowsEmitter
from gehtp_b200.wtop import OP, ROWS_AUTO, Engine
from test_f32_rows import f32_bits


def _with_bad_token(mt, value):
    """The model with one more token, whose embedding is `value` throughout."""
    cfg, t = dict(mt[0], vocab=mt[0]["vocab"] + 1), dict(mt[1])
    t["embed"] = np.concatenate([t["embed"], np.full((1, cfg["width"]), value, np.float32)])
    return cfg, t


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("past,rows,bad", [(0, 16, 5), (0, 8, 1), (61, 20, 12), (64, 7, 6)])
def test_latent_rows_before_a_bad_token(cuda, value, past, rows, bad):
    """fp32 latent attention: rows of a run in front of a token whose latent is no number."""
    mt = _with_bad_token(rip.make([rip.latent(heads=2, dim=24, rot_dim=16, vdim=19, kv_rank=300, ff=None)], seed=9), value)
    tok = rip.ids(past + bad, seed=past + bad)
    want = ripidra_oracle.run(*mt, tok)[0][past:, :-1]
    s = rip.session(cuda, mt, "float32", max_tokens=128)
    if past:
        s.feed(tok[:past], [0])
    got = s.feed(tok[past:] + [mt[0]["vocab"] - 1] * (rows - bad), range(bad))
    s.close()
    assert rip.close(got[:, :-1], want, "float32")


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("bad", [1, 6, 7, 17])
def test_delta_rows_before_a_bad_token(cuda, value, bad):
    """Channel-decay recurrence: tokens of a block of four in front of one that is no number."""
    mt = _with_bad_token(rip.make([rip.delta(heads=2, kv_heads=2, dim=128, vdim=40, ff=None)], seed=bad, slow=2.0), value)
    tok = rip.ids(bad, seed=bad)
    want = ripidra_oracle.run(*mt, tok)[0][:, :-1]
    for dtype in rip.DTYPES:
        s = rip.session(cuda, mt, dtype, max_tokens=64)
        got = s.feed(tok + [mt[0]["vocab"] - 1] * 5, range(bad))
        s.close()
        assert rip.close(got[:, :-1], want, dtype), dtype


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads", [(6, 2), (2, 2), (8, 1)])
def test_window_keys_with_scores_of_minus_infinity(cuda, heads, kv_heads):
    """fp32 window attention: keys whose scores are -inf fill a warp's positions, or are the last a row sees."""
    cfg, t = sup.make([sup.layer(heads=heads, kv_heads=kv_heads, ff=None)], seed=heads)
    at, w, H, G = 20, 5, heads, kv_heads                          # a component the rotation leaves alone; a component of the input
    marked = cfg["vocab"] - 1
    t["embed"][:, w] = 0.0
    t["embed"][marked, w] = 4.0
    t["l0.norm1.b"][w], t["l0.norm1"][w] = 0.0, 1.0
    q, k = (t["l0.mix." + n].reshape(r, 24, -1) for n, r in (("q", H), ("k", G)))
    q[:, at], k[:, at], k[:, at, w] = 0.0, 0.0, -100.0            # 0 for every token but the marked one
    t["l0.mix.q.b"].reshape(H, 24)[:, at], t["l0.mix.k.b"].reshape(G, 24)[:, at] = 1.0, 0.0
    t["l0.mix.q.norm"][at], t["l0.mix.k.norm"][at] = 1.0, 3e38    # its key: -sqrt(24) 3e38
    tok = [i % (marked - 1) for i in sup.ids(44, seed=2)]
    for p in (8, 9, 10, 11, 21, 32, 33, 34, 35, 36, 37, 43):
        tok[p] = marked
    want = supevik_oracle.run(cfg, t, tok)[0]
    s = sup.session(cuda, (cfg, t), "float32", max_tokens=64)
    for cut in ([44], [9, 1, 1, 10, 23], [12, 20, 1, 1, 1, 9]):
        assert sup.close(sup.run_cut(s, tok, cut), want, "float32"), cut
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("K,N", [(264, 66), (3072, 130)])
def test_infinite_weights(cuda, K, N):
    """fp32 projection: weights of +-inf against x of few and of many bits, of either sign, and zero (no number then). Bound of
    the finite sums: every one of the K products and sums rounds by at most 2^-24 of what has been added up (2^-23 where
    the tensor core truncates)."""
    rng = np.random.default_rng(K)
    scale = np.float32(1 / 3)
    tab = bf16_to_f32(f32_to_bf16(rng.standard_normal((150, K)).astype(np.float32)))
    tab[:, 9] = np.resize(np.float32([1.0, -2.0, 0.5, 0.0, -1.0, 2.0, -0.5, 0.0]), 150)
    tab[::2, 9] *= 3.0                                            # times scale: one bit in every other row, all 24 in the rest
    w = bf16_to_f32(f32_to_bf16(rng.standard_normal((N, K)).astype(np.float32)))
    w[3, 9], w[64, 9], w[N - 1, 9], w[5, 9], w[5, K - 1] = np.inf, -np.inf, np.inf, np.inf, -np.inf
    e = RowsEmitter("float32", 256, 150, 1)
    t, ws = e.slot("t", lambda: f32_bits(tab)), e.slot("w", lambda: f32_bits(w))
    e.embed(t, 150, K, scale=scale)
    e.op(OP.LINEAR, [e.temp("x"), ws, e.temp("y"), ROWS_AUTO, K, N, 0, 0, 0, 0])
    eng = Engine(cuda, e.finish())
    face = np.zeros(151, np.int32)
    face[:150] = np.arange(150)
    x = (tab * scale).astype(np.float32).astype(np.float64)
    with np.errstate(invalid="ignore"):
        want, size = np.stack([(x * w[n].astype(np.float64)).sum(1) for n in range(N)], 1), np.abs(x) @ np.abs(np.where(np.isinf(w), 0, w)).T.astype(np.float64)
    for rows in (2, 16, 17, 64, 150):
        eng.set_rows(rows, 1)
        eng.run_io(face, e.temp("y"), None)
        got = eng.temp(e.temp("y"), np.float32).reshape(rows, N).astype(np.float64)
        fine = np.isfinite(want[:rows])
        assert np.array_equal(got[~fine], want[:rows][~fine], equal_nan=True), rows
        assert (np.abs(got[fine] - want[:rows][fine]) <= (K + 2) * 2.0 ** -23 * size[:rows][fine]).all(), rows
    eng.shutdown()
