"""The fused path at the ends of what its enclosures cover, against an engine that makes
every bundle in FP64 (CVL_NO_ENCLOSURES): the same counts, chains and info bits. Each case
asserts from the stage names that the ordinary engine did run the fused kernels."""
import numpy as np
import pytest

import curvelet_construction_on_gpu_b200 as cvl
from curvelet_construction_on_gpu_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engines():
    with pytest.MonkeyPatch.context() as m:
        m.setenv("CVL_NO_ENCLOSURES", "1")
        fp64 = cvl.Engine()
    fused = cvl.Engine()
    fused.set_graphs(False)  # stage by stage, so that the stages can be told
    yield fused, fp64
    fused.close()
    fp64.close()


def _stages(eng):
    return {name for name, _ in eng.kernel_times()}


def _assert_fused(eng):
    s = _stages(eng)
    assert "curvelets" in s and "bundles" not in s, s


def _same(a, b):
    for name in ("valid_pairs", "total_neighbor_pairs", "max_num_of_neighbors", "truncated_anchors", "num_curvelets"):
        assert getattr(a, name) == getattr(b, name), name
    assert np.array_equal(a.chains, b.chains)
    assert np.array_equal(np.asarray(a.info).view(np.int64), np.asarray(b.info).view(np.int64))


def _scatter(n, size, seed):
    rng = np.random.default_rng(seed)
    return np.column_stack([rng.uniform(0, size, (n, 2)), rng.uniform(-np.pi, np.pi, n), np.ones(n)])


@pytest.mark.parametrize("nrad", [0.5, 3.5])
@pytest.mark.parametrize("rad,window,edges,size", [(8.0, 8, 30000, 600), (40.0, 8, 30000, 600), (40.0, 32, 6000, 1000)])
def test_search_radius_apart_from_nrad(engines, rad, window, edges, size, nrad):
    """Staged calls, whose neighbour lists have a radius of their own."""
    fused, fp64 = engines
    e = _scatter(edges, size, 3)
    p = cvl.CurveletParams(nrad=nrad)
    got, want = (eng.build_neighbor_graph(e, rad, window, 128) for eng in engines)
    n = fused.form_pairwise_bundles(got, p)
    _assert_fused(fused)
    assert n == fp64.form_pairwise_bundles(want, p) > 0
    r = fused.build_curvelets(got, p)
    _assert_fused(fused)
    _same(r, fp64.build_curvelets(want, p))


def _map(kind):
    if kind == "small":
        return synth.plain_small(3)
    if kind == "lines":  # parallel lines 0.8 to 0.9 px apart: e1 near 0, perpendicular denominators
        gx, k = np.meshgrid(np.arange(200.0), np.arange(12.0))
        return np.column_stack([gx.ravel(), (10 + 0.8 * k + 0.002 * k * k).ravel(), (1e-9 * k).ravel(), np.ones(gx.size)])
    return _scatter(20000, 220, 8)


@pytest.mark.parametrize("turns", [0, 16, 159, 166000])  # orientations within 2 pi, of about 100, 1000 and 1e6 rad
@pytest.mark.parametrize("over", [dict(), dict(max_k=0.002), dict(max_k=2.0 ** -10), dict(max_k=900.0), dict(dx=0.36),
                                  dict(dx=0.36, max_k=2.0 ** -10), dict(nrad=60.0), dict(nrad=1e3), dict(nrad=1e200),
                                  dict(nrad=1e-3)],
                         ids=lambda o: "-".join(f"{k}{v:g}" for k, v in o.items()) or "default")
@pytest.mark.parametrize("kind", ["small", "lines", "scatter"])
def test_angles_and_curvatures(engines, kind, over, turns):
    fused, fp64 = engines
    e = _map(kind).copy()
    e[:, 2] += 2 * np.pi * np.random.default_rng(4).integers(-turns, turns + 1, len(e))
    p = cvl.CurveletParams(**over)
    r = fused.run(e, p)
    _assert_fused(fused)
    _same(r, fp64.run(e, p))


@pytest.mark.parametrize("edges", [517, None])  # both graphs' buckets
def test_orientations_out_of_range(engines, edges):
    """Beyond 2^20 rad the two-kernel path runs, by its own graph where graphs are on."""
    direct, fp64 = engines
    e = (synth.plain_small(3)[:edges] if edges else synth.plain_hd(1000)).copy()
    e[len(e) // 2, 2] += 2 * np.pi * 400_000
    want = fp64.run(e)
    _same(direct.run(e), want)
    assert "bundles" in _stages(direct)
    g = direct.build_neighbor_graph(e)
    assert direct.form_pairwise_bundles(g, cvl.CurveletParams()) == want.valid_pairs
    with cvl.Engine() as eng:
        for k in range(1, 4):
            _same(eng.run(e), want)
            assert _stages(eng) <= {"graph", "start"}, _stages(eng)
            st = eng.graph_stats()
            assert (st["replays"], st["fallbacks"]) == (2 * k, k)
        assert st["captures"] == 3  # (the second graph's buffers make the first be captured again, once)
        plain = e[: len(e) // 2]
        _same(eng.run(plain), fp64.run(plain))  # the next run is not held back
        assert eng.graph_stats()["replays"] == 7
        a, b = eng.run_maps([plain, e])
        _same(a, fp64.run(plain))
        _same(b, want)
