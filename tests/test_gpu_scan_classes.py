"""That the cluster-major scan runs, and with which visits, in the situations whose results the route tests
compare: its three kernels are launched, visits without a candidate, visits whose warmup passes the
first step (heavy ones, computed ahead by the warps of the grid in units of two horizontal blocks), and
heavy visits past the columns that a batch gets (128 vectors a query, at least 32,768)."""
import os
import tempfile

import numpy as np
import pytest

from pdx_b200 import compiled
from pdx_b200.builder import GaussianMixture, build_index

pytestmark = pytest.mark.gpu


def _run(itype, d, n, nlist, comps, nq, k, nprobe, eps0):
    import torch
    gm = GaussianMixture(d, comps, 0.25, seed=3 + d, unit_norm=True)
    f = build_index(gm.sample(n, 0), itype, num_clusters=nlist, num_meso_clusters=5 if "tree" in itype else 0,
                    normalize=True, seed=5)
    path = os.path.join(tempfile.mkdtemp(), "ix.pdx")
    f.save(path)
    ix = compiled.load_index(path)
    ix.set_nprobe(nprobe)
    ix.set_pruning_aggressiveness(eps0)
    q = torch.from_numpy(ix.prepare_queries(gm.sample(nq, 1))).cuda()
    ids = torch.empty(nq, k, dtype=torch.int32, device="cuda")
    dist = torch.empty(nq, k, device="cuda")
    cnt = torch.empty(nq, dtype=torch.int32, device="cuda")
    launches = []
    for mode in (1, 0):
        ix.set_scan_mode(mode)
        ix.search_device(q.data_ptr(), nq, k, ids.data_ptr(), dist.data_ptr(), cnt.data_ptr(), transformed=True,
                         stats=True)
        torch.cuda.synchronize()
        launches.append(ix.last_launch_count())
    assert launches[1] == launches[0] + 3
    return ix.last_scan_stats()


@pytest.mark.parametrize("itype", ["pdx_u8", "pdx_f32"])
def test_heavy_visits(itype):
    assert _run(itype, 256, 6_000, 40, 8, 47, 20, 12, 1.5)["visits_full_warmup"] > 0


@pytest.mark.parametrize("itype", ["pdx_u8", "pdx_tree_f32"])
def test_visits_without_candidates(itype):
    s = _run(itype, 768, 2_000, 30, 60, 300, 10, 9, 1.5)
    assert s["visits_first_step_exit"] > s["candidates"]


@pytest.mark.parametrize("itype", ["pdx_u8", "pdx_f32"])
def test_heavy_visits_without_room(itype):
    nq = 40
    s = _run(itype, 64, 18_000, 2, 2, nq, 10, 2, 1e30)  # every vector of a visit is a candidate
    assert s["visits_full_warmup"] == nq
    assert s["candidates"] > 4 * max(128 * nq, 32768)
