"""A filtered batch in which some queries have no filter, on a tree index whose dimension the tiled top
level cannot take (d not a multiple of 4), with that form asked for (top-level mode 3): the batch is
searched, as it is in every other mode. Batches without a filter stay refused in mode 3."""
import os
import tempfile

import numpy as np
import pytest

from pdx_b200 import compiled
from pdx_b200.builder import GaussianMixture, build_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [5, 40])
def test_mixed_filtered_batch_runs_where_the_tiled_form_cannot(nq):
    d, n, k = 42, 1500, 10
    gm = GaussianMixture(d, 20, 0.4, seed=3, unit_norm=True)
    f = build_index(gm.sample(n, 0), "pdx_tree_u8", num_clusters=30, num_meso_clusters=4, normalize=True, seed=3)
    path = os.path.join(tempfile.mkdtemp(), "ix.pdx")
    f.save(path)
    ix = compiled.load_index(path)
    ix.set_nprobe(9)
    R = ix.prepare_queries(gm.sample(nq, 1))
    rng = np.random.default_rng(7)
    lists = [None if i % 2 else np.flatnonzero(rng.random(n) < 0.3).astype(np.uint64) for i in range(nq)]
    out = []
    for mode in (1, 3):
        ix.set_top_level_mode(mode)
        out.append(ix.filtered_search_batch(R, k, lists, transformed=True))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    with pytest.raises(RuntimeError):
        ix.search_batch(R, k, transformed=True)
