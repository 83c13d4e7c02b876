"""k_curvelets decides on single-precision enclosures and settles the rest in FP64: an
engine that makes every bundle in FP64 (CVL_NO_ENCLOSURES) gives the same counts, chains
and info bits, on ordinary maps and where enclosures are hard put (ties, parallel edges,
dense clusters, close pairs, angles and grids outside their range)."""
import numpy as np
import pytest

import curvelet_construction_on_gpu_b200 as cvl
from curvelet_construction_on_gpu_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fp64_engine():
    with pytest.MonkeyPatch.context() as m:
        m.setenv("CVL_NO_ENCLOSURES", "1")
        eng = cvl.Engine()
    yield eng
    eng.close()


def _rows(x, y, th):
    x, y, th = np.broadcast_arrays(np.asarray(x, float), y, th)
    return np.ascontiguousarray(np.column_stack([x.ravel(), y.ravel(), th.ravel(), np.ones(x.size)]))


def _map(kind):
    rng = np.random.default_rng(5)
    base = synth.plain_small(3)
    if kind == "small":
        return base
    if kind == "reversed":
        return np.ascontiguousarray(base[::-1])
    if kind == "wide_rows":  # edge_data_sz 6, far from the origin
        return np.ascontiguousarray(np.column_stack([base[:, 0] - 3.0e6, base[:, 1] + 1.0e6, base[:, 2:],
                                                     np.zeros((len(base), 2))]))
    if kind == "cluster":  # runs of more than 32 pairs, up to the 128-candidate cap
        return _rows(rng.uniform(0, 14, 700), rng.uniform(0, 14, 700), rng.normal(0.4, 0.3, 700))
    if kind == "band":  # 30-60 neighbours each
        return _rows(rng.uniform(0, 300, 4000), rng.uniform(0, 12, 4000), rng.normal(0.0, 0.4, 4000))
    if kind == "lattice":  # exact ties everywhere
        gx, gy = np.meshgrid(np.arange(40.0), np.arange(30.0))
        return _rows(gx, gy, (gx.astype(int) % 3) * (np.pi / 4))
    if kind == "lines":  # parallel lines 0.8 to 0.9 px apart: e1 near 0, perpendicular denominators
        gx, k = np.meshgrid(np.arange(200.0), np.arange(12.0))
        return _rows(gx, 10 + 0.8 * k + 0.002 * k * k, 1e-9 * k)
    if kind == "duplicates":  # close pairs, coincident edges
        d = np.repeat(base[:800], 2, axis=0)
        d[1::2, :2] += rng.choice([0.0, 0.3, 0.7999999, 0.8000001], (800, 1)) * [1.0, 0.0]
        return np.ascontiguousarray(d)
    if kind == "angles":  # orientations beyond the enclosures' range
        e = base.copy()
        e[::7, 2] += 2.0 * np.pi * 400
        return e
    return synth.mixed_map(2005)  # above 64 Ki edges


KINDS = ["small", "reversed", "wide_rows", "cluster", "band", "lattice", "lines", "duplicates", "angles", "mixed"]


def _same(a, b):
    for name in ("valid_pairs", "total_neighbor_pairs", "max_num_of_neighbors", "truncated_anchors", "num_curvelets"):
        assert getattr(a, name) == getattr(b, name), name
    assert np.array_equal(a.chains, b.chains)
    assert np.array_equal(np.asarray(a.info).view(np.int64), np.asarray(b.info).view(np.int64))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("graphs", [True, False])
def test_same_bits_as_fp64(engine, fp64_engine, kind, graphs):
    e = _map(kind)
    engine.set_graphs(graphs)
    try:
        _same(engine.run(e), fp64_engine.run(e))
    finally:
        engine.set_graphs(True)


@pytest.mark.parametrize("over", [dict(group_max_sz=2), dict(group_max_sz=3), dict(group_max_sz=7), dict(group_max_sz=16),
                                  dict(max_k=0.002), dict(max_k=4.0), dict(nrad=6.0, max_candidates=128),
                                  dict(max_candidates=9), dict(dt_deg=8.0), dict(dt_deg=22.0), dict(dx=0.8, sx=0.2),
                                  dict(sx=0.2), dict(st=0.05), dict(max_candidates=200), dict(dx=0.9, sx=0.225)],
                         ids=lambda d: "-".join(f"{k}{v}" for k, v in d.items()))
@pytest.mark.parametrize("kind", ["small", "band", "lines"])
def test_same_bits_with_other_parameters(engine, fp64_engine, over, kind):
    p = cvl.CurveletParams(**over)
    e = _map(kind)
    _same(engine.run(e, p), fp64_engine.run(e, p))


@pytest.mark.parametrize("kind", ["cluster", "band", "small"])
def test_same_bits_on_a_fresh_engine(fp64_engine, kind):
    """The first run's pair buffers are a guess: a map with more pairs goes again."""
    e = _map(kind)
    with cvl.Engine() as eng:
        eng.set_graphs(False)
        _same(eng.run(e), fp64_engine.run(e))
        _same(eng.run(e), fp64_engine.run(e))
        _same(eng.run(e[: len(e) // 2]), fp64_engine.run(e[: len(e) // 2]))


def test_same_bits_batched_and_staged(engine, fp64_engine):
    maps = [_map(k) for k in ("small", "cluster", "lattice", "angles", "lines")]
    for maps_ in (maps, maps[:3] + maps[4:]):  # with and without a map outside the certified angles
        got, want = engine.run_maps(maps_), fp64_engine.run_maps(maps_)
        for a, b in zip(got, want):
            _same(a, b)
    for m in maps:
        g = engine.build_neighbor_graph(m)
        assert engine.form_pairwise_bundles(g, cvl.CurveletParams()) == \
            fp64_engine.form_pairwise_bundles(fp64_engine.build_neighbor_graph(m), cvl.CurveletParams())


@pytest.mark.parametrize("gms", [2, 3, 4, 7, 16])
@pytest.mark.parametrize("kind", ["band", "lattice", "lines"])
def test_general_path_against_the_oracle(fp64_engine, oracle, kind, gms):
    """k_growth, which leaves out the seeds of the first seed's chain: chains that fill up
    (gms 3, 4) and that do not, runs of ties and of one seed."""
    e = _map(kind)
    r = fp64_engine.run(e, cvl.CurveletParams(group_max_sz=gms))
    o = oracle.run(e, nthreads=4, group_max_sz=gms)
    assert (r.num_curvelets, r.valid_pairs) == (o.num_curvelets, o.valid_pairs)
    assert np.array_equal(r.chains, o.chains)


@pytest.mark.parametrize("run_edges", [0, 70000])
@pytest.mark.parametrize("block_edges", [1, 7, 8, 9, 31, 32, 33, 40, 65])
def test_search_items(engine, fp64_engine, block_edges, run_edges):
    """Hash blocks (8 x 8 px) of as many edges as k_search's items hold (8, on runs of more than
    64 Ki edges 32), one more and one less, apart and side by side, against the two-pass search."""
    rng = np.random.default_rng(block_edges)
    blocks = np.array([(b, r) for r in range(6) for b in range(12) if (b + r) % 3])
    xy = (blocks[:, None, :] * 8 + rng.uniform(-0.45, 7.45, (len(blocks), block_edges, 2))).reshape(-1, 2)
    e = _rows(xy[:, 0], xy[:, 1], rng.normal(0.3, 0.3, len(xy)))
    if run_edges:  # single edges elsewhere
        k = np.arange(run_edges)
        e = np.concatenate([e, _rows(200.0 + 5 * (k % 300), 200.0 + 5 * (k // 300), 0.0)])
    _same(engine.run(e), fp64_engine.run(e))
