"""DELTA_CHUNK ops that carry one state, gathered into one pass over the chunks, against the one-kernel-per-op plan (scalar
sums in the reference's order): head sizes, more rows than a chunk has, operands from slots and from constant windows, what
lies between the chunks, and runlists that must keep their order because memory is shared."""
import numpy as np
import pytest

from conftest import assert_fp16_close
from gehtp_b200.wtop import OP, ST, BlobBuilder, Engine, S


def _operands(rng, H, rows, D):
    k = rng.standard_normal((H, rows, D)).astype(np.float32)
    k = (k / np.linalg.norm(k, axis=-1, keepdims=True)).astype(np.float16)
    v, q = (rng.standard_normal((H, rows, D)).astype(np.float16) for _ in range(2))
    beta = (1 / (1 + np.exp(-rng.standard_normal((H, rows))))).astype(np.float16)
    g = np.log(1 / (1 + np.exp(-rng.standard_normal((H, rows))))).astype(np.float16)
    return k, v, q, beta, g


def _run(cuda, blob, temps, fusion, runs, x):
    cuda.gehtp_cuda_set_fusion(fusion)
    cuda.wt_exec_state_reset()
    eng = Engine(cuda, blob)
    out = []
    for _ in range(runs):
        eng.run_io(x, temps[-1], None)
        out.append([eng.temp(t, np.uint16).copy() for t in temps])
    launches = cuda.gehtp_cuda_launch_count()
    eng.run_io(x, temps[-1], None)
    launches = cuda.gehtp_cuda_launch_count() - launches
    eng.shutdown()
    cuda.gehtp_cuda_set_fusion(1)
    return out, launches


@pytest.mark.gpu
@pytest.mark.parametrize("H,D,n,ntok,q_raw,shared", [(1, 64, 2, 64, 0, ""), (3, 128, 5, 64, 0, ""), (2, 128, 3, 80, 1, ""), (2, 64, 33, 64, 0, ""),
                                                     (2, 128, 3, 64, 0, "result"), (2, 128, 3, 64, 0, "operand")])
def test_delta_run_against_op_by_op(cuda, H, D, n, ntok, q_raw, shared):
    """Three runs that carry the state on (eager, captured, replayed). shared: two chunks write one temp, or a chunk reads
    what an op between the chunks writes - such lists keep one launch per chunk."""
    rng = np.random.default_rng(H + D + n)
    b = BlobBuilder()
    face = b.add_ext_in(64)
    b.add_states([H * D * D * 4])
    b.add_op(OP.UNARY, [S(face), 1, 32, 14])
    temps, tid = [], 2
    for c in range(n):
        args = [S(b.add_slot(a)) for a in _operands(rng, H, ntok, D)]
        if shared == "operand" and c == n - 1:
            args[1] = temps[-1]                                  # v of the last chunk: the transposed result of the one before
        y = 2 if shared == "result" else tid
        b.add_op(OP.DELTA_CHUNK, args + [y, ST(0), 64, ntok, H, D, q_raw])
        b.add_op(OP.TRANSPOSE_GEN, [y, tid + 1, 3, H, ntok, D, 1, 1 | 0 << 8 | 2 << 16])
        temps.append(tid + 1)
        tid += 2
    blob = b.build()
    x = rng.standard_normal(32).astype(np.float16)
    got, launches = _run(cuda, blob, temps, 1, 3, x)
    want, _ = _run(cuda, blob, temps, 0, 3, x)
    assert (launches == 1 + 2 + n) == (not shared)
    rows = np.arange(ntok) < 64                                  # rows past the chunk are not written
    for r in range(3):
        for c in range(n):
            sel = (slice(None),) if shared == "operand" and ntok == 64 else rows
            assert_fp16_close(got[r][c].view(np.float16).reshape(ntok, H, D)[sel], want[r][c].view(np.float16).reshape(ntok, H, D)[sel], "run %d chunk %d" % (r, c))


@pytest.mark.gpu
@pytest.mark.parametrize("H,D,chunks,hidden", [(2, 128, 2, 128), (4, 64, 5, 384), (16, 128, 9, 1024)])
def test_projection_of_all_chunks(cuda, H, D, chunks, hidden):
    """The layer's out-projections run as one GEMM over blocks of 64 rows that lie apart in memory: every chunk's output
    against the one-kernel-per-op plan, an odd number of blocks among them (half of the last tile is missing)."""
    from gehtp_b200.runlists import build_gdn_runlist
    blob, man = build_gdn_runlist(64 * chunks, hidden, 256, 4, H, D, 64)
    x = np.random.default_rng(4).standard_normal((64 * chunks, hidden)).astype(np.float16)
    temps = [man["conv_temp"]] + man["chunk_out"]
    got, launches = _run(cuda, blob, temps, 1, 3, x)
    want, _ = _run(cuda, blob, temps, 0, 3, x)
    assert launches <= 7                                         # two projections (each with a reduction), convolution, the two of the rule
    for r in range(3):
        for c, t in enumerate(temps):
            assert_fp16_close(got[r][c].view(np.float16), want[r][c].view(np.float16), "run %d temp %d" % (r, t))
