"""The tcgen05 GEMMs where a CTA walks several tiles, so that one tile's products start while the accumulator of the one in
front of it is drained: every tile shape, on integers (every order of the sums gives the same fp32 value)."""
import math
import os
import re

import numpy as np
import pytest

from gehtp_b200.checkpoint import f32_to_bf16
from gehtp_b200.rowlists import RowsEmitter
from gehtp_b200.wtop import LIN_X_BF16, LIN_Y_BF16, OP, ROWS_AUTO, Engine

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gehtp_b200", "csrc")
SMS = 148
# (M, K, N): rows and columns of the tile
W4 = {(100, 192, 38016): (128, 128), (300, 512, 25344): (128, 192), (300, 640, 31616): (128, 256), (700, 320, 15872): (256, 128),
      (1000, 1024, 28544): (256, 160), (700, 1024, 25344): (256, 192), (1000, 1024, 23808): (256, 256)}
F16 = {(300, 192, 18944): (128, 128), (300, 192, 31616): (128, 192), (300, 320, 37888): (128, 256), (1000, 2560, 23680): (256, 160),
       (700, 2560, 25216): (256, 192)}


def _choice(w4, M, K, N):
    """(rows, columns, runs of K, tiles) by the cost table of the source and the rule beside it, on 148 SMs."""
    text = open(os.path.join(CSRC, "w4a16_gemm_sm100.cu" if w4 else "f16_gemm_sm100.cu")).read()
    table = [(128 * int(a), int(b), float(c), float(d)) for a, b, c, d in re.findall(r"\{(\d), (\d+), ([\d.]+)f, ([\d.]+)f\}", text)]
    assert len(table) == (7 if w4 else 5)
    G, best = math.ceil(K / 64), None
    for rows, cols, kb, epi in table:
        tiles = math.ceil(M / rows) * math.ceil(N / cols)
        for c in range(1, min(32, G) + 1):
            if c > 1 and (G % c or G // c < (4 if w4 else 6) or 4 * c * M * N > 64 << 20):
                continue
            rounds = math.ceil(tiles * c / SMS)
            if w4:
                rounds = 0.89 * rounds + 0.11 * max(1.0, tiles * c / SMS)
            us = rounds * (G // c * kb + epi)
            if c > 1:
                us += 1.6 + 8 * c * M * N / 7e6 if w4 else 2 + 8 * c * M * N / 5e6
            if best is None or us < best[0] * (0.97 if w4 else 1):
                best = us, rows, cols, c, tiles
    return best[1:]


def test_shapes_give_every_tile():
    for shapes in (W4, F16):
        for (M, K, N), tile in shapes.items():
            *got, runs, tiles = _choice(shapes is W4, M, K, N)
            assert tuple(got) == tile and runs == 1 and tiles > 2 * SMS, (M, K, N)      # some CTA starts its third tile


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,N", [*W4, *F16])
def test_many_tiles_exact_on_integers(cuda, M, K, N):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(M + 3 * K + 7 * N)
    a = torch.randint(-4, 5, (M, K), device="cuda", generator=g).half()
    q = torch.randint(0, 16, (K, N), device="cuda", generator=g, dtype=torch.uint8)
    w = ((q.float() - 8) * 0.25).half()
    want = (a.double() @ w.double()).half()
    y = torch.full((M + 1, N), 7.0, device="cuda").half()              # one row more: nothing is written behind the last
    if (M, K, N) in W4:
        scales = torch.full((K // 64, N), 0.25, device="cuda").half()
        slot = torch.cat([(q[:, 0::2] | q[:, 1::2] << 4).reshape(-1), scales.view(torch.uint8).reshape(-1)]).contiguous()
        packed = torch.zeros(K * N // 8, device="cuda", dtype=torch.int32)
        torch.cuda.synchronize()
        assert cuda.gehtp_dev_w4_repack(slot.data_ptr(), packed.data_ptr(), K, N) == 0
        rc = cuda.gehtp_dev_w4a16_matmul(a.data_ptr(), packed.data_ptr(), scales.data_ptr(), y.data_ptr(), M, K, N, 2)
    else:
        wt = w.T.contiguous()
        torch.cuda.synchronize()
        rc = cuda.gehtp_dev_matmul_f16_nk(a.data_ptr(), wt.data_ptr(), y.data_ptr(), M, K, N)
    assert rc == 0 and cuda.gehtp_cuda_sync() == 0, cuda.gehtp_cuda_last_error()
    assert torch.equal(y[:M], want) and (y[M] == 7.0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,N", list(F16))
def test_many_tiles_with_bf16_rows(cuda, M, K, N):
    """bf16 rows of a row-count runlist: bf16 and fp32 results."""
    import torch
    rng = np.random.default_rng(N)
    tab = rng.integers(-4, 5, (M, K)).astype(np.float32)
    w = np.resize(rng.integers(-8, 8, (997, K)).astype(np.float32) * np.float32(0.25), (N, K))
    want = (torch.from_numpy(tab).cuda().double() @ torch.from_numpy(w[:997]).cuda().double().T).float().cpu().numpy()
    want = want[:, np.arange(N) % 997]
    e = RowsEmitter("bfloat16", 256, M, 1)
    t, ws = e.slot("t", lambda: f32_to_bf16(tab)), e.slot("w", lambda: np.resize(f32_to_bf16(w[:997]), (N, K)))
    e.embed(t, M, K)
    e.op(OP.LINEAR, [e.act(), ws, e.temp("f"), ROWS_AUTO, K, N, LIN_X_BF16, 0, 0, 0])
    e.op(OP.LINEAR, [e.act(), ws, e.temp("b"), ROWS_AUTO, K, N, LIN_X_BF16 | LIN_Y_BF16, 0, 0, 0])
    eng = Engine(cuda, e.finish())
    face = np.zeros(M + 1, np.int32)
    face[:M] = np.arange(M)
    eng.set_rows(M, 1)
    eng.run_io(face, e.temp("f"), None)
    assert np.array_equal(eng.temp(e.temp("f"), np.float32).reshape(M, N), want)
    assert np.array_equal(eng.temp(e.temp("b"), np.uint16).reshape(M, N), f32_to_bf16(want))
    eng.shutdown()
