"""GPU parity of filtered search (pdxg_search.cu, the device-built selection bitmaps): selectivities
on both sides of the warmup rule (0.2), filters that pass fewer rows than k, every threads-per-query
form, row ids that repeat, are out of order or do not exist, and float distances at and above the
mask value. The oracle takes the same numbers in the same order: no tolerance."""
import os
import tempfile

import numpy as np
import pytest

from pdx_b200 import compiled
from pdx_b200.builder import GaussianMixture, build_index
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu


def _index(port_cls, itype, d, n, nlist, normalize=True):
    gm = GaussianMixture(d, 20, 0.4, seed=d + 1, unit_norm=normalize)
    f = build_index(gm.sample(n, 0), itype, num_clusters=nlist, num_meso_clusters=4 if "tree" in itype else 0,
                    normalize=normalize, seed=3)
    path = os.path.join(tempfile.mkdtemp(), "ix.pdx")
    f.save(path)
    return compiled.load_index(path), port_cls(path), gm


@pytest.fixture(scope="module")
def port_cls(built_oracle):
    from oracle.oracle import Port
    return Port


@pytest.mark.parametrize("itype,d,nlist", [("pdx_tree_u8", 256, 12), ("pdx_u8", 42, 30), ("pdx_f32", 130, 12),
                                           ("pdx_tree_f32", 64, 25)])
@pytest.mark.parametrize("threads", [0, 64, 256, 512])
def test_selectivities_match_the_oracle(port_cls, itype, d, nlist, threads):
    n = 3000
    ix, port, gm = _index(port_cls, itype, d, n, nlist)
    R = ix.prepare_queries(gm.sample(10, 1))
    rng = np.random.default_rng(7)
    lists = [np.flatnonzero(rng.random(n) < s).astype(np.uint64) for s in (0.002, 0.03, 0.19, 0.21, 0.6, 1.0)]
    lists.append(rng.permutation(np.repeat(lists[1], 3)))                              # repeated, out of order
    lists.append(np.concatenate([lists[2], np.array([n, 2**32 + 5, 2**63], np.uint64)]))  # no such rows
    lists.append(np.zeros(0, np.uint64))
    lists.append(None)
    ix.set_threads_per_query(threads)
    for k in (1, 10, 150):
        for nprobe in (0, 5):
            ix.set_nprobe(nprobe)
            port.set_nprobe(nprobe)
            ids, ds, cnt = ix.filtered_search_batch(R, k, lists, transformed=True)
            for i in range(len(R)):
                if lists[i] is None:
                    pi, pd = port.search(R[i], k, transformed=True)
                else:
                    # the engine counts a repeated row once; the oracle takes each row once
                    pi, pd = port.filtered_search(R[i], k, np.unique(lists[i][lists[i] < n]), transformed=True)
                assert_same(ids[i, :cnt[i]], ds[i, :cnt[i]], pi, pd, ctx=f"{itype} k={k} nprobe={nprobe} list {i}")
    port.close()


def test_distances_above_the_mask_value(port_cls):
    """Selected vectors farther than FLT_MAX / 2: the masked slots come first, as in the reference."""
    d, n = 64, 600
    ix, port, gm = _index(port_cls, "pdx_f32", d, n, 6, normalize=False)
    R = np.zeros((2, d), np.float32)
    R[0, 0], R[1, :] = 1.45e19, 1.7e18
    lists = [np.arange(0, n, 3, dtype=np.uint64)] * 2
    ids, ds, cnt = ix.filtered_search_batch(R, 10, lists, transformed=True)
    for i in range(2):
        pi, pd = port.filtered_search(R[i], 10, lists[i], transformed=True)
        assert_same(ids[i, :cnt[i]], ds[i, :cnt[i]], pi, pd, ctx=f"q{i}")
    port.close()
