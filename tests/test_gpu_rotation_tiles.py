"""GPU rotation by FP32 FMA chains (pdxg_rotate.cu): the 32x32-tile GEMM of small batches gives the
bits of the 128x64-tile GEMM of large ones (the same chain per output; no tolerance), at tile
remainders in rows, columns and K; the few-row form agrees with both at FP32 rounding level: d + 1
roundings of 2^-24 relative to |q||m| = 1 on normalized rows, twice for two forms."""
import os
import tempfile

import numpy as np
import pytest

from pdx_b200 import compiled
from pdx_b200.builder import GaussianMixture, build_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [8, 33, 100, 256])
@pytest.mark.parametrize("normalize", [True, False])
def test_tile_forms_agree(d, normalize):
    gm = GaussianMixture(d, 8, 0.4, seed=d, unit_norm=normalize)
    f = build_index(gm.sample(500, 0), "pdx_f32", num_clusters=5, normalize=normalize, seed=2)
    path = os.path.join(tempfile.mkdtemp(), "ix.pdx")
    f.save(path)
    ix = compiled.load_index(path)
    n = 128 * ((300 + (d + 63) // 64 - 1) // ((d + 63) // 64))  # at least 300 large tiles
    Q = np.random.default_rng(d).standard_normal((n, d)).astype(np.float32)
    large = ix.prepare_queries(Q)
    for m in (9, 31, 33, 65, 130):
        np.testing.assert_array_equal(ix.prepare_queries(Q[:m]), large[:m], err_msg=f"{m} rows")
    scale = 1.0 if normalize else float(np.linalg.norm(Q[:8], axis=1).max())
    for m in (1, 7, 8):
        np.testing.assert_allclose(ix.prepare_queries(Q[:m]), large[:m], rtol=0, atol=2 * (d + 1) * 2.0**-24 * scale,
                                   err_msg=f"{m} rows")
