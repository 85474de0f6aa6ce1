"""Latent attention over many rows with heads of 128 + 64 / 128 (tcgen05): one tile and several, portions behind cached
positions that end inside a tile, scores that let single keys stand out, against the plain statement."""
import numpy as np
import pytest

import ripidra_oracle
import test_ripidra as rip


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
