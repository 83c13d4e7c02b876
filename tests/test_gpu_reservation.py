"""cvl_engine_reserve_workspace on sparse shapes: runs within a reserved shape of a few pairs
per edge allocate no device memory and go through in one pass, kernel by kernel too."""
import numpy as np
import pytest

import curvelet_construction_on_gpu_b200 as cvl

pytestmark = pytest.mark.gpu


def _scatter(n, per_edge, seed):
    """n edges with about per_edge neighbours each (0: none within the radius)."""
    rng = np.random.default_rng(seed)
    if per_edge == 0:
        k = np.arange(n)
        xy = np.column_stack([k % 200, k // 200]) * 6.0
    else:
        xy = rng.uniform(0, np.sqrt(n * np.pi * 3.5 ** 2 / per_edge), (n, 2))
    return np.column_stack([xy, rng.normal(0.3, 0.3, n), np.ones(n)])


def _same(a, b):
    assert np.array_equal(a.chains, b.chains)
    assert np.array_equal(np.asarray(a.info).view(np.int64), np.asarray(b.info).view(np.int64))
    assert (a.valid_pairs, a.total_neighbor_pairs) == (b.valid_pairs, b.total_neighbor_pairs)


@pytest.mark.parametrize("n", [3000, 90000])
@pytest.mark.parametrize("per_edge", [0, 1, 2, 3])
def test_a_sparse_reserved_shape_allocates_nothing(n, per_edge):
    maps = [_scatter(n, per_edge, 1), _scatter(n // 3, per_edge, 2)]
    with cvl.Engine() as grown, cvl.Engine() as eng:
        for x in (grown, eng):
            x.set_graphs(False)
        want = [grown.run(m) for m in maps]
        eng.reserve_workspace(n, max(r.total_neighbor_pairs for r in want), max(r.num_curvelets for r in want))
        m0 = eng.memory()
        for _ in range(2):
            for m, w in zip(maps, want):
                _same(eng.run(m), w)
                stages = [name for name, _ in eng.kernel_times()]
                assert stages.count("curvelets") == 1 and "bundles" not in stages and "neighbors_count" not in stages
        assert eng.memory()["device_grows"] == m0["device_grows"]
        # a run past the reserved pairs still gives its results
        dense = _scatter(n, 12, 3)
        _same(eng.run(dense), grown.run(dense))
        _same(eng.run(maps[0]), want[0])


def test_a_budget_without_room_for_more_pairs():
    """The guess of 32 pairs per edge is not made where the budget has no room for it, and the
    buffers that are there stay."""
    m = _scatter(60000, 2, 4)
    with cvl.Engine() as free:
        free.set_graphs(False)
        want = free.run(m)
    with cvl.Engine() as eng:
        eng.set_graphs(False)
        eng.reserve_workspace(10000, 10000, 10000)
        small = _scatter(10000, 1, 5)
        eng.run(small)
        held = eng.memory()["held_bytes"]
    for extra in (60000 * 300, 60000 * 420, 60000 * 900):  # bytes for the run's other buffers, and a little
        with cvl.Engine(mem_budget_bytes=held + extra) as eng:
            eng.set_graphs(False)
            eng.reserve_workspace(10000, 10000, 10000)
            eng.run(small)
            try:
                _same(eng.run(m), want)
            except cvl.CvlError as ex:
                assert ex.code == cvl._abi.CVL_ENOMEM
            assert eng.memory()["held_bytes"] <= held + extra
            eng.run(small)
