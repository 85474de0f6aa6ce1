"""A session whose run fails: on the device (states between two runs, given back) or before it (states as they were)."""
import numpy as np
import pytest

from gehtp_b200.session import Session
from gehtp_b200.wtop import EngineError


class _Engine:
    """Stands in for the engine; the next run fails with `rc`."""
    rc, resets = 0, 0

    def set_rows(self, rows, sel):
        pass

    def run_io(self, face, out_temp, out):
        if self.rc:
            raise EngineError(self.rc, "failed")
        out[:] = 7.0

    def state_reset(self):
        self.resets += 1


@pytest.mark.parametrize("rc,position,resets", [(-1, 0, 2), (3, 2, 1)])
def test_failed_run(rc, position, resets):
    s = object.__new__(Session)
    s.engine, s.vocab = _Engine(), 11
    s.man = dict(vocab=11, max_rows=8, max_sel=2, nslots=16, logits_temp=1)
    s._face = np.zeros(10, np.int32)
    s.reset()
    s.feed([1, 2], want=(1,))
    s.engine.rc = rc
    with pytest.raises(EngineError):
        s.feed([3], want=(0,))
    assert (s.position, s.engine.resets) == (position, resets)
    s.engine.rc = 0
    assert s.feed([4], want=(0,)).shape == (1, 11)
