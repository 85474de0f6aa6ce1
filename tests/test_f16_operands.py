"""fp16 products whose second operand, stored [N, K], is what the op in front of them writes."""
import numpy as np
import pytest

from conftest import assert_fp16_close
from gehtp_b200.wtop import OP, BlobBuilder, Engine, S

K = 512


def _run(cuda, build, out, shape, want, wshape):
    """Runs the blob for operand after operand: the place of the second operand holds the one before."""
    rng = np.random.default_rng(shape[0])
    b = BlobBuilder()
    face = b.add_ext_in(2 * wshape[0] * wshape[1])
    build(b, face, rng)
    eng = Engine(cuda, b.build())
    for _ in range(5):                                            # the last ones replay a captured run
        w = rng.standard_normal(wshape).astype(np.float16)
        eng.run_io(w, out, None)
        assert_fp16_close(eng.temp(out).reshape(shape), want(w.astype(np.float32)))
    eng.shutdown()


@pytest.mark.gpu
@pytest.mark.parametrize("M,N", [(1, 64), (7, 1024), (8, 4096), (31, 200), (33, 256)])
def test_operand_of_the_op_in_front(cuda, M, N):
    x = (np.random.default_rng(M).standard_normal((M, K)) * 0.1).astype(np.float16)

    def build(b, face, rng):
        b.add_op(OP.UNARY, [S(face), 1, N * K, 0])
        b.add_op(OP.MATMUL_F16, [S(b.add_slot(x)), 1, 2, M, K, N, 2])
    _run(cuda, build, 2, (M, N), lambda w: x.astype(np.float32) @ -w.T, (N, K))


@pytest.mark.gpu
@pytest.mark.parametrize("M", [3, 16, 31])
def test_feed_forward_of_operands_of_the_op_in_front(cuda, M):
    N = 320
    x = (np.random.default_rng(M).standard_normal((M, K)) * 0.02).astype(np.float16)

    def build(b, face, rng):
        n, xs = M * N, b.add_slot(x)
        b.add_op(OP.UNARY, [S(face), 1, 2 * N * K, 0])
        b.add_op(OP.SPLIT, [1, 8] + [0] * 7 + [0, 2, N * K, N * K, 0, 0, 0])
        b.add_op(OP.SPLIT, [1, 2] + [0] * 7 + [0, 2, N * K, N * K, 0, 0, 1])
        for op in ([OP.MATMUL_F16, [S(xs), 8, 3, M, K, N, 2]], [OP.UNARY, [3, 4, n, 8]], [OP.BINARY, [3, 4, 5, n, 2]],
                   [OP.MATMUL_F16, [S(xs), 2, 6, M, K, N, 2]], [OP.BINARY, [5, 6, 7, n, 2]]):
            b.add_op(*op)

    def want(w):
        g, u = x.astype(np.float32) @ -w[:N].T, x.astype(np.float32) @ -w[N:].T
        return g / (1 + np.exp(-g)) * u
    _run(cuda, build, 7, (M, N), want, (2 * N, K))


@pytest.mark.gpu
def test_weight_slot_filled_by_an_op_of_the_run(cuda):
    """A slot that a memory-planner op writes is no constant of the run."""
    M, N = 4, 256
    x = (np.random.default_rng(0).standard_normal((M, K)) * 0.1).astype(np.float16)

    def build(b, face, rng):
        pool = b.add_slot(np.zeros((N, K), np.float16))
        b.add_op(OP.UNARY, [S(face), 1, N * K, 0])
        b.add_op(OP.SPILL, [1, pool, 0, N * K])
        b.add_op(OP.MATMUL_F16, [S(b.add_slot(x)), S(pool), 2, M, K, N, 2])
    _run(cuda, build, 2, (M, N), lambda w: x.astype(np.float32) @ -w.T, (N, K))
