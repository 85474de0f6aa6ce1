"""Channel-decay recurrence in chunks of 16 tokens (heads of 128 key channels, runs of 32 rows and more) against the plain
statement: last chunks that are not full, value columns of one CTA and of several, shared keys, runs longer than one window of
scratch, cuts, decays from none to vanishing, values that are no numbers."""
import numpy as np
import pytest

import ripidra_oracle
import test_ripidra as rip
from test_nonfinite_rows import _with_bad_token


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,vdim,slow,cut", [
    (1, 1, 16, 0.0, [32]), (3, 1, 48, 9.0, [33, 47]), (4, 2, 128, -6.0, [95, 32, 3]), (2, 2, 32, 3.0, [1041]), (19, 19, 128, 1.0, [64]),
])
def test_chunked_recurrence(cuda, heads, kv_heads, vdim, slow, cut):
    mt = rip.make([rip.delta(heads=heads, kv_heads=kv_heads, dim=128, vdim=vdim, ff=None)], seed=heads, slow=slow)
    tok = rip.ids(sum(cut), seed=vdim)
    want = ripidra_oracle.run(*mt, tok)[0]
    for dtype in rip.DTYPES:
        s, got, at = rip.session(cuda, mt, dtype, max_tokens=1100), [], 0
        for n in cut:
            got.append(s.feed(tok[at:at + n], range(n)))
            at += n
        s.close()
        assert rip.close(np.concatenate(got), want, dtype), dtype


@pytest.mark.gpu
@pytest.mark.parametrize("cut", [[31, 32, 33], [63, 64], [65, 16]])
def test_lines_between_the_forms(cuda, cut):
    """9 heads (72 CTAs) change to chunks at 32 rows, 19 heads (152 CTAs) at 64."""
    for heads in (9, 19):
        mt = rip.make([rip.delta(heads=heads, kv_heads=heads, dim=128, vdim=128, ff=None)], seed=heads, slow=1.0)
        tok = rip.ids(sum(cut), seed=cut[0])
        want = ripidra_oracle.run(*mt, tok)[0]
        s, got, at = rip.session(cuda, mt, "bfloat16", max_tokens=256), [], 0
        for n in cut:
            got.append(s.feed(tok[at:at + n], range(n)))
            at += n
        s.close()
        assert rip.close(np.concatenate(got), want, "bfloat16"), heads


@pytest.mark.gpu
@pytest.mark.parametrize("cut", [[490, 3], [497, 2, 500]])
def test_convolution_at_the_line_between_one_and_two_channels_a_thread(cuda, cut):
    """7296 channels: 899 CTAs of one channel a thread at 496 rows and more."""
    mt = rip.make([rip.delta(heads=19, kv_heads=19, dim=128, vdim=128, ff=None)], seed=4, slow=1.0)
    tok = rip.ids(sum(cut), seed=cut[0])
    want = ripidra_oracle.run(*mt, tok)[0]
    for dtype in rip.DTYPES:
        s, got, at = rip.session(cuda, mt, dtype, max_tokens=1024), [], 0
        for n in cut:
            got.append(s.feed(tok[at:at + n], [0, 1, n - 1]))
            at += n
        s.close()
        at = np.cumsum([0] + cut[:-1])
        assert rip.close(np.concatenate(got), np.concatenate([want[[a, a + 1, a + n - 1]] for a, n in zip(at, cut)]), dtype), dtype


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("rows,bad", [(32, 1), (40, 39), (60, 23), (50, 16)])
def test_rows_in_front_of_a_bad_token(cuda, value, rows, bad):
    mt = _with_bad_token(rip.make([rip.delta(heads=2, kv_heads=1, dim=128, vdim=32, ff=None)], seed=bad, slow=2.0), value)
    tok = rip.ids(rows, seed=bad)
    want = ripidra_oracle.run(*mt, tok[:bad])[0][:, :-1]
    for dtype in rip.DTYPES:
        s = rip.session(cuda, mt, dtype, max_tokens=64)
        got = s.feed(tok[:bad] + [mt[0]["vocab"] - 1] + tok[bad + 1:], range(bad))
        s.close()
        assert rip.close(got[:, :-1], want, dtype), dtype
