"""Chunks of the delta rule whose results take the memory of operands: such lists keep one launch per chunk, since the CTAs
of a gathered run walk the chunks at their own pace."""
import numpy as np
import pytest

from conftest import assert_fp16_close
from gehtp_b200.wtop import OP, ST, BlobBuilder, S
from test_delta_runs import _operands, _run

H, D, CHUNKS = 2, 64, 3


@pytest.mark.gpu
@pytest.mark.parametrize("reader,operand,writer", [(0, 0, 1), (0, 1, 2), (1, 2, 2), (None, 0, 0)])
def test_results_on_operands(cuda, reader, operand, writer):
    """Operand `operand` (k, v, q) of chunk `reader` is a temp made in front of the run, the result of chunk `writer` goes by
    its id. reader None: ids of their own, the run is gathered."""
    rng = np.random.default_rng(operand + 3 * writer)
    data = [list(_operands(rng, H, 64, D)) for _ in range(CHUNKS)]
    b = BlobBuilder()
    face = b.add_ext_in(64)
    b.add_states([H * D * D * 4])
    b.add_op(OP.UNARY, [S(face), 1, 32, 14])
    shared = 2
    args = [[S(b.add_slot(a)) for a in chunk] for chunk in data]
    if reader is not None:
        b.add_op(OP.UNARY, [S(b.add_slot(-data[reader][operand])), shared, H * 64 * D, 0])
        args[reader][operand] = shared
    temps = []
    for c in range(CHUNKS):
        y = shared if reader is not None and c == writer else 10 + c
        b.add_op(OP.DELTA_CHUNK, args[c] + [y, ST(0), 64, 64, H, D, 0])
        b.add_op(OP.TRANSPOSE_GEN, [y, 20 + c, 3, H, 64, D, 1, 1 | 0 << 8 | 2 << 16])
        temps.append(20 + c)
    x = rng.standard_normal(32).astype(np.float16)
    got, launches = _run(cuda, b.build(), temps, 1, 3, x)
    want, _ = _run(cuda, b.build(), temps, 0, 3, x)
    assert launches == (1 + 2 + CHUNKS if reader is None else 2 + 2 * CHUNKS)
    for r in range(3):
        for c in range(CHUNKS):
            assert_fp16_close(got[r][c].view(np.float16), want[r][c].view(np.float16), "run %d chunk %d" % (r, c))
