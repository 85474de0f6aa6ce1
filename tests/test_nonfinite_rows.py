"""Values that are not finite: a row's result holds nothing of tokens behind it, and infinite scores and weights count as in
plain fp32 arithmetic, however kernels cut rows, keys and sums."""
import numpy as np
import pytest

import ripidra_oracle
import test_ripidra as rip


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
