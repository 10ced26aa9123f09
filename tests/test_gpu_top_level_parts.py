"""GPU parity of the tiled tree top level (pdxg_toplevel.cu) over its forms: stages of a tile in one
CTA or shared by several (small batches), and the replay's heap in one register a lane (k up to 32),
four (128) or shared memory. The visit orders and the results equal those of the per-query top-level
kernel (mode 2), which takes the same decisions on the same floats: no tolerance."""
import os
import tempfile

import numpy as np
import pytest

from pdx_b200 import compiled
from pdx_b200.builder import GaussianMixture, build_index

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(64, 9), (260, 12), (768, 5)])
def index(request):
    d, nmeso = request.param
    gm = GaussianMixture(d, 150, 0.3, seed=d, unit_norm=True)
    f = build_index(gm.sample(6000, 0), "pdx_tree_u8", num_clusters=300, num_meso_clusters=nmeso, normalize=True,
                    seed=4)
    path = os.path.join(tempfile.mkdtemp(), "ix.pdx")
    f.save(path)
    ix = compiled.load_index(path)
    return ix, ix.prepare_queries(gm.sample(5000, 1))


@pytest.mark.parametrize("nq", [1, 7, 200, 5000])
@pytest.mark.parametrize("nprobe", [1, 32, 33, 128, 129, 0])
def test_tiled_top_level_equals_the_per_query_form(index, nq, nprobe):
    import torch
    ix, R = index
    q = torch.from_numpy(R[:nq].copy()).cuda()
    ix.set_nprobe(nprobe)
    out = []
    for mode in (0, 2):
        ix.set_top_level_mode(mode)
        ids = torch.empty(nq, 10, dtype=torch.int32, device="cuda")
        d = torch.empty(nq, 10, device="cuda")
        cnt = torch.empty(nq, dtype=torch.int32, device="cuda")
        ix.search_device(q.data_ptr(), nq, 10, ids.data_ptr(), d.data_ptr(), cnt.data_ptr(), transformed=True)
        torch.cuda.synchronize()
        orders, counts = ix.last_visit_orders(nq, nprobe or 300)
        rows = [orders[i, :counts[i]].tolist() for i in range(nq)]
        out.append((rows, ids.cpu().numpy(), d.cpu().numpy(), cnt.cpu().numpy()))
    ix.set_top_level_mode(0)
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1:], out[1][1:]):
        np.testing.assert_array_equal(a, b)
