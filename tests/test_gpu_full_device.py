"""Searches on a device whose memory is nearly used up: the arrays of the batched Start, the scan and the
centroid probe shrink to what there is, and a tree's top level takes the form without partials
(pdxg_index.cu). Results stay the same, the batch can still be captured, and with the memory free again
the next search takes its whole batch at once."""
import numpy as np
import pytest

from pdx_b200 import compiled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("itype,d,nlist,nprobe", [("pdx_f32", 16, 10, 0), ("pdx_u8", 16, 10, 0),
                                                  ("pdx_tree_f32", 128, 1000, 64)])  # 0.9 GB of partials
def test_arrays_shrink_to_the_free_memory(itype, d, nlist, nprobe):
    import torch
    n, nq, k = 20_000, 60_000, 10
    rng = np.random.default_rng(5)
    ix = compiled.PDXIndex(itype, d, seed=11, num_clusters=nlist, num_meso_clusters=32 if "tree" in itype else 0,
                           normalize=False)
    ix.build_index(rng.standard_normal((n, d)).astype(np.float32))
    ix.set_nprobe(nprobe)
    q = torch.from_numpy(ix.prepare_queries(rng.standard_normal((nq, d)).astype(np.float32))).cuda()
    ids = torch.empty(nq, k, dtype=torch.int32, device="cuda")
    dist = torch.empty(nq, k, device="cuda")
    cnt = torch.empty(nq, dtype=torch.int32, device="cuda")

    def run(index, m=nq, graph=False):
        args = (q.data_ptr(), m, k, ids.data_ptr(), dist.data_ptr(), cnt.data_ptr())
        if graph:
            index.capture(*args, transformed=True).launch(0)
        else:
            index.search_device(*args, transformed=True)
        torch.cuda.synchronize()
        return [x.cpu().numpy().copy() for x in (ids, dist, cnt)]

    run(ix, 3000)  # the kernels of every route are loaded
    ix.set_scan_mode(1)
    ix.set_start_mode(1)
    ix.set_top_level_mode(2)
    expect = run(ix)  # the per-query route: its buffers are there from now on
    ix.set_scan_mode(0)
    ix.set_start_mode(0)
    ix.set_top_level_mode(0)
    torch.cuda.empty_cache()
    filler = []
    for keep in (8 << 30, 160 << 20):
        size = torch.cuda.mem_get_info()[0] - keep
        if size > 0:
            filler.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
    try:
        for graph in (False, True):
            for a, b in zip(run(ix, graph=graph), expect):
                np.testing.assert_array_equal(a, b)
            sliced = ix.last_launch_count()
    finally:
        del filler
        torch.cuda.empty_cache()
    for a, b in zip(run(ix), expect):
        np.testing.assert_array_equal(a, b)
    assert ix.last_launch_count() < sliced


def test_a_search_after_a_refused_one():
    """A batch whose results have no room is refused; the next search does not report that again."""
    import torch
    n, d = 2_000, 16
    rng = np.random.default_rng(6)
    ix = compiled.PDXIndex("pdx_f32", d, seed=11, num_clusters=10, normalize=False)
    ix.build_index(rng.standard_normal((n, d)).astype(np.float32))
    ix.set_nprobe(0)
    q = rng.standard_normal((200_000, d)).astype(np.float32)
    expect = ix.search_batch(q[:64], 10)
    torch.cuda.empty_cache()
    filler = []
    for keep in (8 << 30, 160 << 20):
        size = torch.cuda.mem_get_info()[0] - keep
        if size > 0:
            filler.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
    try:
        with pytest.raises(RuntimeError):
            ix.search_batch(q, 300)  # 480 MB of results
        for a, b in zip(ix.search_batch(q[:64], 10), expect):
            np.testing.assert_array_equal(a, b)
    finally:
        del filler
        torch.cuda.empty_cache()
