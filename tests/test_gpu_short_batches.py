"""Which batches of short pairs stay out of tiles, at the edges of the rule, and that both kernels give
the oracle's results there. The number of resident warps tells the kernels apart: the one-score kernel
has up to 32 an SM, one a pair; the tile kernel 16 a block."""
import numpy as np
import pytest

import biwfa_gpu_pii2025_gb300 as pkg
from oracle import binding

pytestmark = pytest.mark.gpu
AFFINE, EDIT, INDEL, LINEAR = binding.METRIC_AFFINE, binding.METRIC_EDIT, binding.METRIC_INDEL, binding.METRIC_LINEAR
PEN = {AFFINE: (0, 4, 6, 2), EDIT: (0, 1, 0, 0), INDEL: (0, 1, 0, 0), LINEAR: (0, 4, 2, 0)}


def _batch(groups, seed):
    """groups: (pairs, plen + tlen); texts are the patterns with two substitutions, one longer if odd."""
    rng = np.random.default_rng(seed)
    seqs, plen, tlen = [], [], []
    for n, total in groups:
        a, b = total // 2, total - total // 2
        p = rng.choice(np.frombuffer(b"ACGT", np.uint8), (n, a))
        t = np.concatenate([p, np.full((n, b - a), ord("T"), np.uint8)], axis=1)
        for _ in range(2):
            t[np.arange(n), rng.integers(0, b, n)] = rng.choice(np.frombuffer(b"ACGT", np.uint8), n)
        seqs.append(np.concatenate([p, t], axis=1).reshape(-1))
        plen += [a] * n
        tlen += [b] * n
    plen, tlen = np.array(plen, np.int32), np.array(tlen, np.int32)
    start = np.concatenate([[0], np.cumsum(plen.astype(np.int64) + tlen)])[:-1]
    return pkg.PairBatch(np.concatenate(seqs), start, plen, start + plen, tlen)


@pytest.mark.parametrize("metric,score_only,groups,tiles", [
    (AFFINE, False, [(16384, 136)], False), (AFFINE, False, [(16384, 137)], True), (AFFINE, False, [(16383, 136)], True),
    (AFFINE, True, [(16384, 112)], False), (AFFINE, True, [(16384, 113)], True),
    (AFFINE, True, [(65536, 170)], False), (AFFINE, True, [(65536, 171)], True),
    (AFFINE, False, [(65536, 184)], False), (AFFINE, False, [(65536, 185)], True),
    (AFFINE, False, [(65480, 80), (64, 350)], False), (AFFINE, False, [(65480, 80), (65, 350)], True),
    (AFFINE, False, [(65480, 80), (64, 370)], True),
    (LINEAR, False, [(8192, 204)], False), (LINEAR, False, [(8192, 205)], True), (LINEAR, False, [(8191, 204)], True),
    (LINEAR, False, [(8130, 80), (64, 280)], False), (LINEAR, False, [(8130, 80), (65, 280)], True),
    (LINEAR, True, [(8192, 204)], True),
    (EDIT, False, [(6000, 256)], False), (EDIT, True, [(6000, 256)], False), (EDIT, False, [(6000, 257)], True),
    (EDIT, False, [(16384, 1000)], False), (EDIT, False, [(16384, 1001)], True), (EDIT, True, [(16384, 1000)], True),
    (EDIT, True, [(65536, 1000)], False), (EDIT, True, [(65536, 1001)], True),
    (INDEL, False, [(65030, 80), (512, 1600)], False), (INDEL, False, [(65030, 80), (513, 1600)], True),
    (INDEL, False, [(65030, 80), (512, 1640)], True)])
def test_short_batches_at_the_rules_edges(batch_aligner, metric, score_only, groups, tiles):
    b = _batch(groups, 5)
    res = batch_aligner.align(b, penalties=PEN[metric], metric=metric, score_only=score_only)
    assert (batch_aligner.stats().num_warps <= 2432) == tiles
    assert (res.status == 0).all()
    at = np.concatenate([np.arange(0, b.n, b.n // 1500), np.arange(b.n - 100, b.n)])
    for i in at:
        _, score, ops, _ = binding.oracle_align(b.pattern(i), b.text(i), PEN[metric], score_only, metric=metric)
        assert res.scores[i] == score, i
        assert score_only or pkg.runs_to_ops(res.runs_of(i)) == ops, i
