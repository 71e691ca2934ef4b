"""Leaves of short, very unequal pairs in batches of nothing longer: their leaf store is sized from
the pair itself, and rows in tiles have to fit it. One pair a batch, against the oracle."""
import numpy as np
import pytest

import biwfa_gpu_pii2025_gb300 as pkg
from oracle import binding

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric,pen", [
    (binding.METRIC_LINEAR, (0, 1, 4, 0)), (binding.METRIC_LINEAR, (0, 2, 8, 0)), (binding.METRIC_LINEAR, (0, 3, 4, 0)),
    (binding.METRIC_LINEAR, (0, 4, 1, 0)), (binding.METRIC_AFFINE, (0, 4, 6, 2)), (binding.METRIC_AFFINE, (0, 2, 3, 1))])
def test_unequal_short_pairs_fit_their_leaf_store(batch_aligner, metric, pen):
    rng = np.random.default_rng(7)
    shapes = [(1, 100), (1, 85), (2, 97), (3, 90), (5, 100), (11, 100), (4, 9), (1, 1), (100, 100), (100, 1)]
    for pl, tl in shapes:
        for unlike in (True, False):
            p, t = (b"A" * pl, b"C" * tl) if unlike else (bytes(rng.choice(list(b"ACGT"), n).astype(np.uint8)) for n in (pl, tl))
            res = batch_aligner.align(pkg.PairBatch.from_lists([p], [t]), penalties=pen, metric=metric)
            _, score, ops, _ = binding.oracle_align(p, t, pen, metric=metric)
            assert res.status[0] == 0 and pkg.runs_to_ops(res.runs_of(0)) == ops and res.scores[0] == score, (pl, tl, unlike)
