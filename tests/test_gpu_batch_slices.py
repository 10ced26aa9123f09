"""Batches past a limit of the batched Start or of the cluster-major scan (8 GB of bitmaps, 16-bit chunk
numbers of the Start's work items) go through both in slices (pdxg_index.cu): the kernels of at least
two slices are launched, and results equal the per-query kernel's bit for bit, with filters and with
per-request k and nprobe too."""
import numpy as np
import pytest

from pdx_b200 import compiled

pytestmark = pytest.mark.gpu

# a slice: at least 3 kernels of the batched Start, 3 of the scan, the per-query one
TWO_SLICES = 2 * (3 + 3 + 1)


def _index(itype, d, n, nlist, big=0):
    rng = np.random.default_rng(d + n)
    x = rng.standard_normal((n, d)).astype(np.float32)
    if big:  # one far cluster of this many rows
        x[:big] = 20 * x[0] + 0.2 * rng.standard_normal((big, d)).astype(np.float32)
    ix = compiled.PDXIndex(itype, d, seed=11, num_clusters=nlist, num_meso_clusters=12 if "tree" in itype else 0,
                           normalize=False)
    ix.build_index(x)
    return ix, rng


def _both_routes(ix, run):
    got = run()
    launches = ix.last_launch_count()
    ix.set_scan_mode(1)
    ix.set_start_mode(1)
    expect = run()
    ix.set_scan_mode(0)
    ix.set_start_mode(0)
    for a, b in zip(got, expect):
        np.testing.assert_array_equal(a, b)
    return launches


def test_bitmaps_past_their_limit():
    ix, rng = _index("pdx_f32", 16, 24_000, 1000, big=4000)
    ix.set_nprobe(0)
    q = ix.prepare_queries(rng.standard_normal((20_000, 16)).astype(np.float32))
    assert _both_routes(ix, lambda: ix.search_batch(q, 10, transformed=True)) >= TWO_SLICES


@pytest.mark.parametrize("itype", ["pdx_f32", "pdx_tree_f32"])
def test_work_items_past_their_limit(itype):
    import torch
    n, d, nq, k = 4000, 8, 140_001, 20
    ix, rng = _index(itype, d, n, 600)
    ix.set_nprobe(16)
    R = ix.prepare_queries(rng.standard_normal((nq, d)).astype(np.float32))
    assert _both_routes(ix, lambda: ix.search_batch(R, k, transformed=True)) >= TWO_SLICES

    lists = [None] * nq
    for i in range(0, nq, 997):
        lists[i] = np.flatnonzero(rng.random(n) < 0.1).astype(np.uint64)
    _both_routes(ix, lambda: ix.filtered_search_batch(R, k, lists, transformed=True))

    q = torch.from_numpy(R).cuda()
    filters = [ix.register_filter(np.flatnonzero(rng.random(n) < s).astype(np.uint64)) for s in (0.05, 0.5)]
    table = compiled.request_table(nq)
    table["k"] = rng.choice([3, 10, 20], nq)
    table["nprobe"] = rng.choice([4, 16], nq)
    table["filter_id"] = np.where(rng.random(nq) < 0.02, np.asarray(filters)[rng.integers(0, 2, nq)], -1)
    ctx = compiled.Context(ix)

    def requests():
        ids = torch.empty(nq, k, dtype=torch.int32, device="cuda")
        dist = torch.empty(nq, k, device="cuda")
        cnt = torch.empty(nq, dtype=torch.int32, device="cuda")
        ctx.search_requests(q.data_ptr(), nq, table, None, k, ids.data_ptr(), dist.data_ptr(), cnt.data_ptr(),
                            transformed=True)
        torch.cuda.synchronize()
        return ids.cpu().numpy(), dist.cpu().numpy(), cnt.cpu().numpy()

    _both_routes(ix, requests)
