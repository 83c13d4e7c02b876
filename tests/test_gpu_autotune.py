"""The autotuner times the knobs that the batch's path reads, and no others."""
import pytest

import curvelet_construction_on_gpu_b200 as cvl
from curvelet_construction_on_gpu_b200 import synth

pytestmark = pytest.mark.gpu


def _tune(eng, m, params):
    before = eng.get_tuning(1)
    b = eng.upload_batch([m])
    try:
        t, ms = eng.autotune(b, params)
    finally:
        b.close()
    assert ms > 0 and eng.get_tuning(1) == t
    return before, t


def test_fused_runs_keep_their_tuning():
    with cvl.Engine() as eng:
        before, after = _tune(eng, synth.plain_hd(1000), cvl.CurveletParams())
        st = eng.graph_stats()
        assert after == before
        assert (st["captures"], st["replays"]) == (1, 4)  # the present tuning, timed


def test_other_grids_are_searched():
    with cvl.Engine() as eng:
        _tune(eng, synth.plain_hd(1000), cvl.CurveletParams(sx=0.2))
        assert eng.graph_stats()["captures"] > 5
