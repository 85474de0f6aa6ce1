"""Prefill attention on scores that stand out: row maxima that later key tiles raise by far, rows that see keys of every other tile
only, infinite scores and values that are no numbers, against the one-kernel-per-op plan."""
import numpy as np
import pytest

from conftest import assert_fp16_close
from gehtp_b200.runlists import Emitter
from gehtp_b200.wtop import Engine, S

NH, KVH = 4, 2


def _attend(cuda, q, k, v, mask):
    """[seq, NH * hd] of the fused plan and of the op-by-op plan. q [seq, NH, hd], k and v [seq, KVH, hd]."""
    seq, _, hd = q.shape
    e = Emitter()
    q, k, v, m = (S(e.b.add_slot(a.astype(np.float16))) for a in (q, k, v, mask))
    mask_b = e.broadcast(m, (1, 1, seq, seq), (1, NH, seq, seq))
    scale_b = e.broadcast(e.const_f16(hd ** -0.5), (1, 1, 1, 1), (1, 1, 1, NH * seq * seq))
    qh, kh, vh = e.transpose3(q, (seq, NH, hd), (1, 0, 2)), e.transpose3(k, (seq, KVH, hd), (1, 2, 0)), e.transpose3(v, (seq, KVH, hd), (1, 0, 2))
    s = e.binary(e.bmm(qh, kh, KVH, NH // KVH * seq, hd, seq), scale_b, NH * seq * seq, 2)
    p = e.softmax(e.binary(s, mask_b, NH * seq * seq, 0), NH * seq, seq)
    out = e.transpose3(e.bmm(p, vh, KVH, NH // KVH * seq, seq, hd), (NH, seq, hd), (1, 0, 2))
    res = []
    for fusion in (1, 0):
        cuda.gehtp_cuda_set_fusion(fusion)
        eng = Engine(cuda, e.b.build())
        eng.run()
        assert (cuda.gehtp_cuda_fused_ops() >= 9) == bool(fusion)
        res.append(eng.temp(out).reshape(seq, NH, hd).astype(np.float64))
        eng.shutdown()
    cuda.gehtp_cuda_set_fusion(1)
    return res


def _inputs(seq, hd, seed):
    rng = np.random.default_rng(seed)
    mask = np.where(np.tril(np.ones((seq, seq), bool)), 0.0, -np.inf)
    return [rng.standard_normal((seq, n, hd)) for n in (NH, KVH, KVH)] + [mask]


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("growth", [3.0, 1 / 3.0])
def test_maxima_that_later_tiles_raise(cuda, hd, growth):
    q, k, v, mask = _inputs(700, hd, 1)
    k *= (growth ** (np.arange(700) // 128 - (0 if growth > 1 else 5)))[:, None, None]
    got, want = _attend(cuda, q, k, v, mask)
    for r0 in range(0, 700, 128):
        assert_fp16_close(got[r0:r0 + 128], want[r0:r0 + 128], "rows from %d" % r0)


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [128, 64])
def test_rows_alive_in_every_other_tile(cuda, hd):
    q, k, v, mask = _inputs(520, hd, 2)
    r, c = np.arange(520)[:, None], np.arange(520)[None, :]
    mask = np.where((r % 3 == 2) | (c // 128 % 2 == r % 3), 0.0, -np.inf)
    got, want = _attend(cuda, q, k, v, mask)
    for i in range(3):
        assert_fp16_close(got[i::3], want[i::3], "rows of kind %d" % i)


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("seq,at", [(100, 3), (300, 40), (300, 200)])
def test_values_that_are_no_numbers(cuda, hd, seq, at):
    """Rows from the first that holds or sees such a value (in front of it the op chain adds it to the mask). An fp16 result that is no
    number is an infinity."""
    for name, value in (("q", np.nan), ("k", np.nan), ("k", np.inf), ("v", np.nan)):
        q, k, v, mask = _inputs(seq, hd, at)
        dict(q=q, k=k, v=v)[name][at, 0, 5] = value
        got, want = (a[at:] for a in _attend(cuda, q, k, v, mask))
        bad = ~np.isfinite(want)
        assert bad.any() and not bad.all() and np.array_equal(bad, ~np.isfinite(got)), (name, value)
        assert_fp16_close(got[~bad], want[~bad], name)


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("row,at", [(90, 3), (250, 100), (299, 130)])
def test_scores_beyond_fp16(cuda, hd, row, at):
    """One score of one row is +inf: inf - inf, no number in all of the row; the others are large."""
    q, k, v, mask = _inputs(300, hd, row)
    k[at, 0] = 2000.0 * np.sign(q[row, 0])
    got, want = (a[at:] for a in _attend(cuda, q, k, v, mask))
    bad = ~np.isfinite(want)
    assert bad[row - at, 0].all() and np.array_equal(bad, ~np.isfinite(got))
    assert_fp16_close(got[~bad], want[~bad])
