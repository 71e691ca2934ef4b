"""The train step's gradient at the edges of its tiles and grid, against the float64 oracle."""
import numpy as np
import pytest

import biwfa_gpu_pii2025_gb300 as pkg
from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def aligner():
    al = pkg.BatchAligner(0)
    yield al
    al.close()


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 152 * 16, 152 * 16 + 1, 5000])
def test_gradient_at_tile_and_grid_edges(aligner, rows):
    """The train step's tiles of 16 rows and its grid of one block per SM: a lone row, both sides of a
    tile and of the grid. Tolerances are test_gradient_matches_float64_oracle's."""
    b = pkg.PairBatch.generate(2, rows, seed=64)
    aligner.upload(b)
    pred = pkg.ScorePredictor(aligner, seed=12)
    try:
        rng = np.random.default_rng(6)
        params = (rng.standard_normal(mo.N_PARAMS) * 0.2).astype(np.float32)
        pred.set_params(params)
        X = mo.bf16_bits_to_float(pred.features())
        t = rng.uniform(0, 8, b.n).astype(np.float32)
        loss, g = pred.gradient(t)
        loss_ref, g_ref = mo.loss_and_grad(params.astype(np.float64), X, t.astype(np.float64))
        assert abs(loss - loss_ref) <= 1e-3 * max(1.0, abs(loss_ref))
        assert np.linalg.norm(g - g_ref) <= 1e-3 * np.linalg.norm(g_ref)
    finally:
        pred.close()
