"""The step count that a batch's run reports: whole chunks of 32 up to the one in
which the last scenario ended, at most the caller's limit."""
import pytest

import slab
from test_blocks import CFG, DX, Z, _release

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("totals,limit,want", [((0.1,), None, 32), ((0.32,), None, 32), ((0.33,), None, 64), ((0.05, 0.4), None, 64),
                                               ((0.4,), 20, 20), ((0.4,), 40, 40), ((0.1,), 20, 20), ((0.1,), 8, 8)])
def test_run_counts_whole_chunks(totals, limit, want):
    b = slab.Batch(Z, DX, max_scenarios=4)
    for k, t in enumerate(totals):
        b.add_release(dict(CFG, total_time=t, output_dt=t), _release(16.0 + 2 * k))
    assert (b.run() if limit is None else b.run(limit)) == want
    if limit is None:
        assert b.run() == 32  # nothing left to do: one chunk that does nothing
    b.close()
