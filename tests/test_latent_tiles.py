"""Latent attention over many rows with heads of 128 + 64 / 128 (tcgen05): one tile and several, portions behind cached
positions that end inside a tile, scores that let single keys stand out, against the plain statement."""
import numpy as np
import pytest

import ripidra_oracle
import test_ripidra as rip
from test_nonfinite_rows import _with_bad_token


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_rank,sharp,cut", [
    (1, 64, 1.0, [40]), (3, 72, 4.0, [128, 129]), (2, 512, 1.0, [100, 57, 300]), (2, 96, 8.0, [513]), (5, 64, 1.0, [127, 1, 200, 33]),
])
def test_rows(cuda, heads, kv_rank, sharp, cut):
    mt = rip.make([rip.latent(heads=heads, dim=128, rot_dim=64, vdim=128, kv_rank=kv_rank, ff=None)], seed=heads, sharp=sharp)
    tok = rip.ids(sum(cut), seed=kv_rank)
    want = ripidra_oracle.run(*mt, tok)[0]
    s, got, at = rip.session(cuda, mt, "bfloat16", max_tokens=640), [], 0
    for n in cut:
        got.append(s.feed(tok[at:at + n], range(n)))
        at += n
    s.close()
    assert rip.close(np.concatenate(got), want, "bfloat16")


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("past,rows,bad", [(0, 96, 1), (0, 96, 95), (0, 200, 127), (0, 200, 128), (150, 200, 120), (1, 40, 17)])
def test_rows_before_a_bad_token(cuda, value, past, rows, bad):
    """Rows of a run in front of a token whose latent is no number, in its tile and in others."""
    mt = _with_bad_token(rip.make([rip.latent(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=72, ff=None)], seed=bad, sharp=2.0), value)
    tok = rip.ids(past + rows, seed=bad)
    tok[past + bad] = mt[0]["vocab"] - 1
    want = ripidra_oracle.run(*mt, tok[:past + bad])[0][past:, :-1]
    s = rip.session(cuda, mt, "bfloat16", max_tokens=640)
    if past:
        s.feed(tok[:past], [0])
    got = s.feed(tok[past:], range(rows))
    s.close()
    assert rip.close(got[:bad, :-1], want, "bfloat16")
    assert not np.isfinite(got[bad:, :-1]).any()
