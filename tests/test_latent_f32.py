"""Latent attention of fp32 rows, eight rows of a head at a time: runs that end inside such a tile and behind a block of 64
keys, ranks of one and of several column groups per thread, against the 64-bit oracle."""
import pytest

import ripidra_oracle as oracle
from test_ripidra import close, ids, latent, make, session

LAYERS = {"rank 40": latent(heads=2, dim=24, rot_dim=16, vdim=19, kv_rank=40, ff=None), "rank 300": latent(heads=3, dim=13, rot_dim=6, vdim=34, kv_rank=300, ff=None),
          "rank 700": latent(heads=1, dim=40, rot_dim=8, vdim=16, kv_rank=700, scale=0.1, ff=None)}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(LAYERS))
def test_tiles_of_eight_rows(cuda, name):
    mt = make([LAYERS[name]], seed=len(name) + 3)
    tok = ids(140, seed=5)
    want = oracle.run(*mt, tok)[0]
    s = session(cuda, mt, "float32", max_tokens=160)
    for cut in ([140], [7, 8, 9, 1, 16, 17, 23], [63, 1, 1, 64, 11]):
        s.reset()
        at = 0
        for n in cut:
            pick = list(range(n))[-64:]                          # at most 64 rows are wanted of one run
            got = s.feed(tok[at:at + n], pick)
            assert close(got, want[at:at + n][pick], "float32"), (cut, at)
            at += n
    s.close()
