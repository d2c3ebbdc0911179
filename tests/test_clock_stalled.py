"""The host clock on a void resident batch (trace status 5 in the first row): the
batch is refused by name, the clock stays and the batch pending."""
import numpy as np
import pytest

from nhflood.clock import STALLED, HostClock


@pytest.mark.parametrize('rows', [1, 32])
def test_stalled_batch_is_refused(rows):
    clock = HostClock(0.0, batch_size=rows)
    clock.begin(10.0, 0.0)
    trace = np.zeros((rows, 10), np.uint32)
    trace[0, 3] = STALLED
    trace[1:, 3] = 1     # rows of steps that some blocks completed
    with pytest.raises(RuntimeError, match='lost one another'):
        clock.read_trace(trace)
    assert clock.pending and clock.now_ticks == 0
