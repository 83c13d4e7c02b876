"""The items of the one-pass search (csrc/cvl_search.cuh), restated: k_bin_scatter lists every
bucket in runs of at most item_size anchors, and k_search ends an item at its head's
bucket, which it hashes from the head's pixel cell. A non-finite edge lies in bucket 0
whatever its cell, so an item that it heads would take other buckets' anchors, each of them
twice (and the wide ones past the end of their list), or none: no items are listed of a run
that holds one, and the curvelet kernels leave it before they read its rows."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "curvelet_construction_on_gpu_b200", "csrc")
M32 = 0xFFFFFFFF


def _hash(bx, by):
    h = ((bx * 73856093) ^ (by * 19349663)) & M32
    h ^= h >> 16
    h = h * 0x7FEB352D & M32
    h ^= h >> 15
    h = h * 0x846CA68B & M32
    return h ^ (h >> 16)


def _processed(cells, finite, item_size, table=1024, seed=0):
    """How often k_search would take each anchor, without its early return."""
    n = len(cells)
    own = np.array([_hash(int(x) >> 3, int(y) >> 3) & (table - 1) for x, y in cells])
    bucket = np.where(finite, own, 0)
    start = np.concatenate([[0], np.cumsum(np.bincount(bucket, minlength=table))])
    pos = np.empty(n, int)  # a bucket's edges take its places in any order
    left = np.bincount(bucket, minlength=table)
    items, at = [], np.empty(n, int)
    for e in np.random.default_rng(seed).permutation(n):
        left[bucket[e]] -= 1
        pos[e] = start[bucket[e]] + left[bucket[e]]
        at[pos[e]] = e
        if left[bucket[e]] & (item_size - 1) == 0:
            items.append(pos[e])
    taken = np.zeros(n, int)
    for c0 in items:
        c1 = min(start[own[at[c0]] + 1], c0 + item_size)
        taken[c0:c1] += 1
    return taken


@pytest.mark.parametrize("item_size", [8, 32])
@pytest.mark.parametrize("edges", [1, 7, 31, 33, 900, 5000])
def test_finite_edges_are_taken_once(item_size, edges):
    cells = np.random.default_rng(edges).integers(0, 60, (edges, 2))
    assert np.all(_processed(cells, np.ones(edges, bool), item_size) == 1)


@pytest.mark.parametrize("item_size", [8, 32])
@pytest.mark.parametrize("cell", [(-2 ** 31, 0), (-2 ** 31, -2 ** 31), (2 ** 31 - 1, 5)])
def test_a_non_finite_head_breaks_the_items(item_size, cell):
    """Why the kernels may not read such a run."""
    cells = np.random.default_rng(1).integers(0, 60, (900, 2))
    cells[400] = cell
    finite = np.arange(900) != 400
    assert any(np.any(_processed(cells, finite, item_size, seed=s) != 1) for s in range(200))


def _kernel(file, name):
    with open(os.path.join(CSRC, file)) as f:
        return re.search(r"__global__ void[^;{]*\b" + name + r"\([^{]*\)\s*\{(.*?)\n\}\n", f.read(), re.S).group(1)


def test_no_items_are_listed_of_such_a_run():
    keys, scatter = _kernel("cvl_kernels.cuh", "k_bin_keys"), _kernel("cvl_kernels.cuh", "k_bin_scatter")
    assert re.search(r"!isfinite\(x\)[^}]*atomicOr\(unfit, UNFIT_NONFINITE\)[^}]*continue;", keys)
    assert "const bool list = items && *unfit == 0u;" in scatter
    assert re.findall(r"if \((.*)\) items\[", scatter)[0].startswith("list && ")


@pytest.mark.parametrize("kernel", ["k_curvelets", "k_curvelets_exact"])
def test_the_curvelet_kernels_leave_such_a_run_first(kernel):
    body = _kernel("cvl_curvelets.cuh", kernel)
    guard = re.search(r"if \(\*a\.unfit\) (return;|\{[^}]*return;)", body)
    reads = re.search(r"a\.(over_list|over_cnt|over_queue|row|csr_ids|F|B)\b", body)
    assert guard and guard.start() < reads.start()
