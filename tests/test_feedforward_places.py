"""Gated feed-forward whose temps share memory, as an offset table or a recycled temp id may lay them once their values are dead,
against the one-kernel-per-op plan."""
import numpy as np
import pytest

from conftest import assert_fp16_close
from gehtp_b200.runlists import dequant_f16, rand_w4
from gehtp_b200.wtop import OP, BlobBuilder, Engine, S

K = 256
X, GATE, SIG, ACT, UP, Y = range(1, 7)


def _blob(quant, rows, N, ids, offsets):
    """x = copy of the input; gate = x Wg; sig; act = gate sig; up = x Wu; y = act up. `offsets`: temp -> place in the table."""
    rng = np.random.default_rng(rows + N)
    b = BlobBuilder()
    x = b.add_slot((rng.standard_normal((rows, K)) * 0.5).astype(np.float16))
    w = []
    for _ in range(2):
        nib, sc = rand_w4(rng, K, N)
        if quant == "w4":
            w.append(b.add_slot(np.concatenate([nib.reshape(-1), sc.view(np.uint8).reshape(-1)]), count=K * N))
        else:
            w.append(b.add_slot(np.ascontiguousarray(dequant_f16(nib, sc).T)))
    n = rows * N
    if offsets:                                                   # entries for temps apart from one another keep their places
        size = {t: 2 * rows * K if t == X else 2 * n for t in offsets}
        b.add_tempoff(max(o + size[t] for t, o in offsets.items()), [(t, o, size[t]) for t, o in offsets.items()], bump_kb=64)
    op, flags = (OP.MATMUL_W4A16, []) if quant == "w4" else (OP.MATMUL_F16, [2])
    b.add_op(OP.UNARY, [S(x), X, rows * K, 14])
    b.add_op(op, [X, S(w[0]), ids[GATE], rows, K, N] + flags)
    b.add_op(OP.UNARY, [ids[GATE], ids[SIG], n, 8])
    b.add_op(OP.BINARY, [ids[GATE], ids[SIG], ids[ACT], n, 2])
    b.add_op(op, [X, S(w[1]), ids[UP], rows, K, N] + flags)
    b.add_op(OP.BINARY, [ids[ACT], ids[UP], ids[Y], n, 2])
    return b.build()


def _check(cuda, quant, rows, N, ids=None, offsets=None, fused=5):
    ids = {**{t: t for t in range(1, 7)}, **(ids or {})}
    blob, out = _blob(quant, rows, N, ids, offsets), []
    for fusion in (1, 0):
        cuda.gehtp_cuda_set_fusion(fusion)
        eng = Engine(cuda, blob)
        eng.run()
        if fusion:
            assert cuda.gehtp_cuda_fused_ops() == fused
        out.append([eng.temp(ids[t]) for t in (UP, Y)])
        eng.shutdown()
    cuda.gehtp_cuda_set_fusion(1)
    assert_fp16_close(out[0][1], out[1][1], "result")
    if quant == "f16" and ids[UP] != ids[Y]:                      # the fp16 forms leave the products readable
        assert_fp16_close(out[0][0], out[1][0], "up projection")


FORMS = [("f16", 3, 512), ("f16", 16, 512), ("f16", 33, 512), ("f16", 128, 512), ("f16", 33, 200), ("w4", 128, 192), ("w4", 128, 256)]


def _far(rows, N):
    """Places of x, and of a product, apart from one another."""
    return lambda i: 2 * rows * K + 4096 + i * (2 * rows * N + 512)


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["whole", "part", "id"])
@pytest.mark.parametrize("quant,rows,N", FORMS)
def test_up_projection_over_the_gate(cuda, quant, rows, N, where):
    at = _far(rows, N)
    if where == "id":
        _check(cuda, quant, rows, N, ids={UP: GATE})
    else:
        shift = 0 if where == "whole" else rows * N // 2 // 8 * 16
        _check(cuda, quant, rows, N, offsets={X: 0, GATE: at(0), UP: at(0) + shift, Y: at(3)})


@pytest.mark.gpu
@pytest.mark.parametrize("quant,rows,N", FORMS)
def test_result_over_the_gate(cuda, quant, rows, N):
    at = _far(rows, N)
    _check(cuda, quant, rows, N, offsets={X: 0, GATE: at(0), UP: at(2), Y: at(0)})
    _check(cuda, quant, rows, N, offsets={X: 0, GATE: at(0), UP: at(3), Y: at(0) + rows * N // 2 // 8 * 16})


@pytest.mark.gpu
@pytest.mark.parametrize("quant,rows,N", FORMS)
def test_one_temp_for_gate_up_and_result(cuda, quant, rows, N):
    _check(cuda, quant, rows, N, ids={UP: GATE, Y: GATE}, fused=5 if (quant, N) == ("w4", 256) else 0)


@pytest.mark.gpu
@pytest.mark.parametrize("quant,rows,N", FORMS + [("w4", 3, 256)])
def test_result_over_the_input(cuda, quant, rows, N):
    """The input is dead behind the up projection; the forms of one launch read it until they are done."""
    at = _far(rows, N)
    _check(cuda, quant, rows, N, offsets={X: 0, GATE: at(0), UP: at(1), Y: 0})
    _check(cuda, quant, rows, N, offsets={X: 512, GATE: at(0), UP: at(1), Y: 0})


@pytest.mark.gpu
@pytest.mark.parametrize("quant,rows,N", FORMS + [("w4", 3, 256)])
def test_one_temp_for_input_and_result(cuda, quant, rows, N):
    _check(cuda, quant, rows, N, ids={Y: X}, fused=0 if (quant, rows) == ("w4", 3) else 5)
