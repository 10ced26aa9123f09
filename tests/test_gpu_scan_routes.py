"""GPU parity of the batched Start and the cluster-major scan (pdxg_start.cu, pdxg_scan.cu): F32
levels (tiles of 8 queries x 64 vectors x 64 dims with remainders in each, unaligned dimensions,
visits without candidates, light and heavy ones, queries that are not finite), and heaps that take
several Starts to fill, or more than are batched. The kernels keep the per-query kernel's chains and their order, so the three routes (cluster-major scan;
per-query kernel after a batched Start; per-query kernel alone) agree bit for bit: no tolerance."""
import os
import tempfile

import numpy as np
import pytest

from pdx_b200 import compiled
from pdx_b200.builder import GaussianMixture, build_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("itype,d,n,nlist,comps,nq,k,nprobe", [
    ("pdx_f32", 64, 18_000, 2, 2, 40, 10, 2),       # no shared-memory bitmaps, one query per CTA
    ("pdx_f32", 33, 3_000, 30, 10, 65, 7, 0),       # unaligned rows, every cluster visited
    ("pdx_f32", 256, 6_000, 40, 8, 47, 20, 12),     # heavy visits
    ("pdx_tree_f32", 130, 3_000, 24, 6, 33, 100, 24),   # d_v not a multiple of 4, heaps near the cluster size
    ("pdx_tree_f32", 768, 2_000, 30, 60, 300, 10, 9),   # several queries per cluster, empty visits
    ("pdx_u8", 96, 3_000, 60, 60, 50, 100, 0),      # heaps of two or three Starts
    ("pdx_tree_u8", 256, 2_000, 100, 30, 33, 150, 50),  # more Starts than are batched: the rest per query
    ("pdx_f32", 8, 4_000, 200, 40, 64, 3, 40),      # fewer dims than the first warmup step
])
@pytest.mark.parametrize("eps0", [1.5, 0.3, 1e30])
def test_three_routes_agree(itype, d, n, nlist, comps, nq, k, nprobe, eps0):
    gm = GaussianMixture(d, comps, 0.25, seed=3 + d, unit_norm=True)
    f = build_index(gm.sample(n, 0), itype, num_clusters=nlist, num_meso_clusters=5 if "tree" in itype else 0,
                    normalize=True, seed=5)
    path = os.path.join(tempfile.mkdtemp(), "ix.pdx")
    f.save(path)
    ix = compiled.load_index(path)
    ix.set_nprobe(nprobe)
    ix.set_pruning_aggressiveness(eps0)
    R = ix.prepare_queries(gm.sample(nq, 1)).copy()
    R[3, d // 2] = np.inf
    R[5, 0] = np.nan
    out = []
    for start, scan in ((0, 0), (0, 1), (1, 1)):
        ix.set_start_mode(start)
        ix.set_scan_mode(scan)
        out.append(ix.search_batch(R, k, transformed=True))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
