"""A run with a non-finite or out-of-range edge is refused (CVL_EINVAL) and leaves
everything else as it was: other batches on the device, and the engine's later runs."""
import numpy as np
import pytest

import curvelet_construction_on_gpu_b200 as cvl
from curvelet_construction_on_gpu_b200 import _abi, synth

pytestmark = pytest.mark.gpu


def _same(a, b):
    assert np.array_equal(a.chains, b.chains)
    assert np.array_equal(np.asarray(a.info).view(np.int64), np.asarray(b.info).view(np.int64))


def _map(kind):
    rng = np.random.default_rng(11)
    if kind == "cluster":  # every anchor's list is cut, or past k_search's columns
        return np.column_stack([rng.uniform(0, 30, 2500), rng.uniform(0, 30, 2500), rng.normal(0.4, 0.3, 2500),
                                np.ones(2500)])
    return synth.plain_small(6) if kind == "small" else synth.mixed_map(2005)


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("kind,max_candidates", [("cluster", 2), ("cluster", 128), ("small", 128), ("small", 2), ("mixed", 2)])
def test_refused_and_nothing_else_changed(kind, max_candidates, graphs):
    e = _map(kind)
    other = synth.plain_small(7)
    p = cvl.CurveletParams(max_candidates=max_candidates)
    n = len(e)
    with cvl.Engine() as eng:
        eng.set_graphs(graphs)
        batch = eng.upload_batch([other, other[:100]])
        good = eng.run(e, p)
        r = eng.run_batch(batch)
        before = [r.take_map(k) for k in range(2)]
        r.close()
        for rows, col, v in (([0], 0, np.nan), ([n // 2], 1, np.inf), ([n - 1], 2, np.nan), ([3], 0, 1.0e9),
                             (range(0, n, 97), 1, -np.inf), (range(n), 2, np.nan)):
            bad = e.copy()
            bad[list(rows), col] = v
            for _ in range(2):
                with pytest.raises(cvl.CvlError) as ei:
                    eng.run(bad, p)
                assert ei.value.code == _abi.CVL_EINVAL
        _same(eng.run(e, p), good)
        r = eng.run_batch(batch)
        for k in range(2):
            _same(r.take_map(k), before[k])
        r.close()
        batch.close()
