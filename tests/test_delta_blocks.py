"""The channel-decay recurrence in blocks of four tokens: head sizes and head counts that lead to each lane layout and CTA
width of its kernel, and runs that end inside a block or a chunk of sixteen, against the 64-bit oracle."""
import numpy as np
import pytest

import ripidra_oracle as oracle
from test_ripidra import DTYPES, close, delta, ids, make, session

LAYERS = {"128 channels": delta(heads=2, kv_heads=2, dim=128, vdim=40, ff=None), "100 channels, odd values": delta(heads=3, kv_heads=1, dim=100, vdim=33, ff=None),
          "70 channels by single copies": delta(heads=2, kv_heads=1, dim=70, vdim=18, ff=None), "76 heads": delta(heads=76, kv_heads=4, dim=68, vdim=32, ff=None)}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(LAYERS))
def test_runs_that_end_inside_a_block(cuda, name):
    mt = make([LAYERS[name]], seed=len(name), slow=2.0)
    tok = ids(57, seed=3)
    want = oracle.run(*mt, tok)[0]
    for dtype in DTYPES:
        s = session(cuda, mt, dtype, max_tokens=64)
        for cut in ([5, 6, 7, 8, 16, 15], [17, 18, 19], [57], [20, 32, 5]):
            s.reset()
            at, rows = 0, []
            for n in cut:
                rows.append(s.feed(tok[at:at + n], range(n)))
                at += n
            assert close(np.concatenate(rows), want[:at], dtype), (dtype, cut)
        s.close()
