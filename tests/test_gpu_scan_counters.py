"""The cluster-major scan's counters (pdxg_get_scan_stats) over its visit classes. With pruning off
every vector of every visit after the Starts is a candidate and a survivor, whichever class the visit
has (unless the first step covers all dims, where the bound is the heap top itself); in every case the
survivors are some of the candidates. Counts are exact."""
import os
import tempfile

import numpy as np
import pytest

from pdx_b200 import compiled
from pdx_b200.builder import GaussianMixture, build_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("itype,d,n,nlist,comps,nq,k", [
    ("pdx_u8", 256, 6_000, 40, 8, 33, 20),     # heavy visits
    ("pdx_f32", 256, 6_000, 40, 8, 47, 20),
    ("pdx_u8", 64, 18_000, 2, 2, 40, 10),      # no bitmaps in shared memory, heavy visits without room
    ("pdx_f32", 64, 18_000, 2, 2, 40, 10),
    ("pdx_u8", 44, 4_000, 200, 40, 64, 3),     # tiny clusters; the warmup is its first step or two
    ("pdx_f32", 8, 4_000, 200, 40, 64, 3),     # fewer vertical dims than the first step
])
def test_counters(itype, d, n, nlist, comps, nq, k):
    import torch
    gm = GaussianMixture(d, comps, 0.25, seed=3 + d, unit_norm=True)
    f = build_index(gm.sample(n, 0), itype, num_clusters=nlist, normalize=True, seed=5)
    path = os.path.join(tempfile.mkdtemp(), "ix.pdx")
    f.save(path)
    ix = compiled.load_index(path)
    ix.set_nprobe(0)
    q = torch.from_numpy(ix.prepare_queries(gm.sample(nq, 1))).cuda()
    ids = torch.empty(nq, k, dtype=torch.int32, device="cuda")
    dist = torch.empty(nq, k, device="cuda")
    cnt = torch.empty(nq, dtype=torch.int32, device="cuda")
    for eps0 in (1e30, 1.5):
        ix.set_pruning_aggressiveness(eps0)
        ix.search_device(q.data_ptr(), nq, k, ids.data_ptr(), dist.data_ptr(), cnt.data_ptr(), transformed=True,
                         stats=True)
        torch.cuda.synchronize()
        stats, scan = ix.last_stats(), list(ix.last_scan_stats().values())
        started = stats["bytes_by_phase"]["start"] // (d * (1 if itype == "pdx_u8" else 4))
        if eps0 == 1e30 and d > 16:
            assert scan[0] == scan[1] == nq * n - started
        assert scan[0] >= scan[1]
