"""GPU parity of the exact centroid probe ahead of the scan (pdxg_probe.cu): tiles of 32 queries x 32
centroids x 64 dims with remainders in each, the d % 8 tail, rows that are not 16-byte aligned, and
the probe of only a batch's filtered queries on a tree. The oracle takes the same floats in the same
order, so results are equal without a tolerance (assert_same: ids as sets among equal distances)."""
import os
import tempfile

import numpy as np
import pytest

from pdx_b200 import compiled
from pdx_b200.builder import GaussianMixture, build_index
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("itype,d,nlist,nq", [
    ("pdx_f32", 33, 1, 1),        # one centroid, an unaligned tail of one dim
    ("pdx_u8", 63, 31, 33),       # plain loads, d % 8 = 7, one query past a tile
    ("pdx_f32", 130, 33, 31),     # plain loads past two stages, one centroid past a tile
    ("pdx_u8", 72, 65, 64),       # a second stage of 8 dims
    ("pdx_tree_u8", 100, 40, 37),
    ("pdx_tree_f32", 256, 33, 5),
])
def test_probe_tiles_match_the_oracle(built_oracle, itype, d, nlist, nq):
    from oracle.oracle import Port
    gm = GaussianMixture(d, 20, 0.4, seed=d, unit_norm=True)
    f = build_index(gm.sample(2000, 0), itype, num_clusters=nlist, num_meso_clusters=5 if "tree" in itype else 0,
                    normalize=True, seed=3)
    path = os.path.join(tempfile.mkdtemp(), "ix.pdx")
    f.save(path)
    ix, port = compiled.load_index(path), Port(path)
    R = ix.prepare_queries(gm.sample(nq, 1))
    rng = np.random.default_rng(d)
    # every third query unfiltered
    lists = [None if i % 3 == 2 else np.flatnonzero(rng.random(2000) < 0.2).astype(np.uint64) for i in range(nq)]
    for nprobe in (0, 1, (nlist + 1) // 2):
        ix.set_nprobe(nprobe)
        port.set_nprobe(nprobe)
        for filtered in (False, True):
            if filtered:
                ids, ds, cnt = ix.filtered_search_batch(R, 10, lists, transformed=True)
            else:
                ids, ds, cnt = ix.search_batch(R, 10, transformed=True)
            for i in range(nq):
                if filtered and lists[i] is not None:
                    pi, pd = port.filtered_search(R[i], 10, lists[i], transformed=True)
                else:
                    pi, pd = port.search(R[i], 10, transformed=True)
                assert_same(ids[i, :cnt[i]], ds[i, :cnt[i]], pi, pd, ctx=f"{itype} nprobe={nprobe} {filtered} q{i}")
    port.close()
