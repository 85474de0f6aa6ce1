"""Projections of fp32 rows at the edges of their kernels' tiles, against float64."""
import numpy as np
import pytest

from gehtp_b200.checkpoint import bf16_to_f32, f32_to_bf16
from gehtp_b200.rowlists import RowsEmitter
from gehtp_b200.wtop import OP, ROWS_AUTO, Engine


@pytest.mark.gpu
@pytest.mark.parametrize("K,N", [(8, 2), (264, 66), (520, 4), (2056, 1028), (3072, 130)])
def test_f32_projection(cuda, K, N):
    """Rows of 24 significant bits against bf16 weights, one row of infinities. Bound: every one of the K products and sums
    of an fp32 chain rounds by at most 2^-24 of what has been added up (2^-23 where the tensor core truncates)."""
    rng = np.random.default_rng(K + N)
    scale = np.float32(1 / 3)
    tab = bf16_to_f32(f32_to_bf16(rng.standard_normal((160, K)).astype(np.float32)))
    w = bf16_to_f32(f32_to_bf16(np.abs(rng.standard_normal((N, K)).astype(np.float32)) + np.float32(0.01)))
    w *= np.where(rng.random((N, K)) < 0.5, -1, 1).astype(np.float32)
    w[:, 0] = np.abs(w[:, 0])
    tab[5, 0] = np.inf
    e = RowsEmitter("float32", 256, 160, 1)
    t, ws = e.slot("t", lambda: f32_bits(tab)), e.slot("w", lambda: f32_to_bf16(w))
    e.embed(t, 160, K, scale=scale)
    e.op(OP.LINEAR, [e.temp("x"), ws, e.temp("y"), ROWS_AUTO, K, N, 0, 0, 0, 0])
    eng = Engine(cuda, e.finish())
    face = np.zeros(161, np.int32)
    face[:160] = np.arange(160)
    x = (tab * scale).astype(np.float64)
    with np.errstate(invalid="ignore"):
        want, size = x @ w.T.astype(np.float64), np.abs(x) @ np.abs(w).T.astype(np.float64)
    for rows in (1, 2, 3, 4, 5, 16, 17, 64, 65, 150):
        eng.set_rows(rows, 1)
        eng.run_io(face, e.temp("y"), None)
        got = eng.temp(e.temp("y"), np.float32).reshape(rows, N)
        fine = np.arange(rows) != 5
        assert (np.abs(got - want[:rows])[fine] <= (K + 2) * 2.0 ** -23 * size[:rows][fine]).all(), rows
        if rows > 5:
            assert (got[5] == np.inf).all(), rows
    eng.shutdown()


def f32_bits(a):
    """bf16 bits of values that bf16 holds, infinities among them."""
    return (np.ascontiguousarray(a, np.float32).view(np.uint32) >> 16).astype(np.uint16)
