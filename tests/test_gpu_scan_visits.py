"""GPU parity of the cluster-major scan's visit classes (pdxg_scan.cu): visits without candidates,
light visits, heavy visits computed ahead by the CTA's warps, heavy visits that find no room, and
clusters too large for a work item's bitmaps in shared memory. The scan must equal the per-query
kernel (scan mode 1) bit for bit: U8 distances are exact integers, so no tolerance is needed."""
import os
import tempfile

import numpy as np
import pytest

from pdx_b200 import compiled
from pdx_b200.builder import GaussianMixture, build_index

pytestmark = pytest.mark.gpu


# comps below nlist split a mixture component over several clusters, whose later visits keep most
# of their vectors: heavy visits. 2 clusters of about 9,000 vectors pass the shared-memory bitmaps.
@pytest.mark.parametrize("d,n,nlist,comps,nq,k,nprobe", [
    (64, 18_000, 2, 2, 40, 10, 2),       # no shared-memory bitmaps, one query per CTA
    (256, 6_000, 40, 8, 33, 20, 12),     # heavy visits, two horizontal blocks short of a group of three
    (1024, 3_000, 24, 6, 47, 5, 24),     # heavy visits over every checkpoint of 256 vertical dims
    (100, 5_000, 30, 200, 1500, 10, 30),  # several queries per CTA, mostly empty and light visits
    (44, 4_000, 200, 40, 64, 3, 40),     # tiny clusters, odd vertical dims
])
@pytest.mark.parametrize("eps0", [1.5, 0.3, 1e30])
def test_visit_classes_equal_the_per_query_kernel(d, n, nlist, comps, nq, k, nprobe, eps0):
    gm = GaussianMixture(d, comps, 0.25, seed=3 + d, unit_norm=True)
    f = build_index(gm.sample(n, 0), "pdx_u8", num_clusters=nlist, normalize=True, seed=5)
    path = os.path.join(tempfile.mkdtemp(), "ix.pdx")
    f.save(path)
    ix = compiled.load_index(path)
    ix.set_nprobe(nprobe)
    ix.set_pruning_aggressiveness(eps0)
    R = ix.prepare_queries(gm.sample(nq, 1))
    out = []
    for mode in (0, 1):
        ix.set_scan_mode(mode)
        out.append(ix.search_batch(R, k, transformed=True))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
