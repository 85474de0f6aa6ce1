"""Gated W4A16 feed-forward of up to 8 rows whose strips outnumber the CTAs that fit the GPU, against the op-by-op plan: rows that
do not fill the tile, one warp and many to a CTA, strips that the grid does not divide."""
import numpy as np
import pytest

from conftest import assert_fp16_close
from gehtp_b200.runlists import Emitter, rand_w4
from gehtp_b200.wtop import Engine, S


@pytest.mark.gpu
@pytest.mark.parametrize("rows,K,N", [(1, 2560, 9728), (3, 2560, 9760), (8, 2560, 5024), (7, 5120, 4880), (2, 5120, 9488), (5, 1280, 19216), (8, 768, 40016), (3, 256, 80016)])
def test_strips(cuda, rows, K, N):
    rng = np.random.default_rng(K + rows)
    e = Emitter()
    x = S(e.b.add_slot((rng.standard_normal((rows, K)) * 0.1).astype(np.float16)))
    gate = e.linear(x, *rand_w4(rng, K, N), rows)
    act = e.binary(gate, e.unary(gate, rows * N, 8), rows * N, 2)
    y = e.binary(act, e.linear(x, *rand_w4(rng, K, N), rows), rows * N, 2)
    blob, out = e.b.build(), []
    for fusion in (1, 0):
        cuda.gehtp_cuda_set_fusion(fusion)
        eng = Engine(cuda, blob)
        eng.run()
        assert cuda.gehtp_cuda_fused_ops() == 5 * fusion
        out.append(eng.temp(y).reshape(rows, N))
        eng.shutdown()
    cuda.gehtp_cuda_set_fusion(1)
    for r in range(rows):
        assert_fp16_close(out[0][r], out[1][r], "row %d" % r)
    assert_fp16_close(out[0][:, -16:], out[1][:, -16:], "last strip")
