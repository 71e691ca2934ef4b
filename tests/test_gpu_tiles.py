"""Rows in tiles (csrc/biwfa_tiles.cuh) against the oracle, bit for bit: wavefronts that end at and
around the tiles' edges, rows that touch an end early (very different lengths, long gaps), pairs
with bytes outside ACGT, every shape, and penalties of the tiles' ratio with other score spacings."""
import numpy as np
import pytest

import biwfa_gpu_pii2025_gb300 as pkg
from biwfa_gpu_pii2025_gb300 import _capi
from oracle import binding

pytestmark = pytest.mark.gpu


def _mutated(rng, p, edits, gap):
    t = list(p)
    for _ in range(edits):
        j, kind, g = int(rng.integers(0, len(t) + 1)), rng.integers(0, 3), int(rng.integers(1, gap + 1))
        if kind == 0:
            t[j:j + g] = []
        elif kind == 1:
            t[j:j] = list(rng.choice(list(b"ACGT"), g))
        elif j < len(t):
            t[j] = int(rng.choice(list(b"ACGT")))
    return bytes(np.array(t, np.uint8))


def _batch(seed):
    rng = np.random.default_rng(seed)

    def seq(n, alphabet=b"ACGT"):
        return bytes(rng.choice(list(alphabet), n).astype(np.uint8))

    pairs = [(b"", b"ACG"), (b"A", b"A"), (b"A", b"C"), (b"ACGT" * 60, b"ACGT" * 60), (seq(700), seq(40)),
             (seq(30), seq(900)), (seq(400), seq(400)), (b"A" * 150, b"A" * 90 + b"C" * 60)]
    for n in (5, 31, 33, 64, 101, 130, 250, 500, 900, 1600):  # edits: wavefronts 0 - 400 diagonals wide
        for edits in (0, 1, 3, n // 20, n // 8):
            p = seq(n, b"ACGT" if edits != 3 else b"ACGTN")
            pairs.append((p, _mutated(rng, p, edits, 1 + edits % 3)))
        p = seq(n)
        pairs.append((p, _mutated(rng, p, 4, 80)))  # long gaps
    return pkg.PairBatch.from_lists([p for p, _ in pairs], [t for _, t in pairs])


@pytest.mark.parametrize("pen,gw,seed", [((0, 4, 6, 2), 1, 1), ((0, 4, 6, 2), 4, 2), ((0, 4, 6, 2), 8, 3),
                                         ((0, 2, 3, 1), 1, 4), ((0, 6, 9, 3), 1, 5), ((0, 14, 21, 7), 8, 6)])
def test_tiles_match_oracle(batch_aligner, pen, gw, seed):
    b = _batch(seed)
    try:
        batch_aligner.set_exec_shape(gw, False)
        res = batch_aligner.align(b, penalties=pen)
        only = batch_aligner.align(b, penalties=pen, score_only=True)
    finally:
        batch_aligner.set_exec_shape(1, False)
    assert (res.status == 0).all()
    for i in range(b.n):
        _, score, ops, _ = binding.oracle_align(b.pattern(i), b.text(i), pen)
        assert pkg.runs_to_ops(res.runs_of(i)) == ops, (i, b.plen[i], b.tlen[i])
        assert res.scores[i] == (score if ops else 0), i
        st, score, _, _ = binding.oracle_align(b.pattern(i), b.text(i), pen, score_only=True)
        assert only.status[i] == st and (st != 0 or only.scores[i] == score), i


@pytest.mark.parametrize("metric,pen,gw,seed", [
    (binding.METRIC_EDIT, (0, 1, 0, 0), 1, 11), (binding.METRIC_EDIT, (0, 1, 0, 0), 8, 12),
    (binding.METRIC_INDEL, (0, 1, 0, 0), 1, 13), (binding.METRIC_LINEAR, (0, 4, 2, 0), 1, 14),
    (binding.METRIC_LINEAR, (0, 4, 6, 0), 4, 15), (binding.METRIC_LINEAR, (0, 9, 12, 0), 1, 16),
    (binding.METRIC_LINEAR, (0, 1, 4, 0), 1, 17)])
def test_one_component_tiles_match_oracle(batch_aligner, metric, pen, gw, seed):
    """One component: rows go on past touched ends, up to edit's wavefronts of 1,000 diagonals."""
    b = _batch(seed)
    if metric == binding.METRIC_EDIT:
        rng = np.random.default_rng(seed)
        far = [(bytes(rng.choice(list(b"ACGT"), n).astype(np.uint8)), bytes(rng.choice(list(b"ACGT"), m).astype(np.uint8)))
               for n, m in ((2500, 2500), (3000, 700))]
        b = pkg.PairBatch.from_lists([b.pattern(i) for i in range(b.n)] + [p for p, _ in far],
                                     [b.text(i) for i in range(b.n)] + [t for _, t in far])
    try:
        batch_aligner.set_exec_shape(gw, False)
        res = batch_aligner.align(b, penalties=pen, metric=metric)
        only = batch_aligner.align(b, penalties=pen, metric=metric, score_only=True)
    finally:
        batch_aligner.set_exec_shape(1, False)
    assert (res.status == 0).all()
    for i in range(b.n):
        _, score, ops, _ = binding.oracle_align(b.pattern(i), b.text(i), pen, metric=metric)
        assert pkg.runs_to_ops(res.runs_of(i)) == ops, (i, b.plen[i], b.tlen[i])
        assert res.scores[i] == (score if ops else 0), i
        st, score, _, _ = binding.oracle_align(b.pattern(i), b.text(i), pen, True, metric=metric)
        assert only.status[i] == st and (st != 0 or only.scores[i] == score), i


@pytest.mark.parametrize("pen,gw,seed", [((0, 4, 6, 2), 1, 21), ((0, 4, 6, 2), 8, 22), ((0, 2, 3, 1), 1, 23)])
def test_wide_searches_match_oracle(batch_aligner, pen, gw, seed):
    """Searches whose two directions meet in blocks of 300 - 1,500 diagonals, whose I and D rows are
    completed only then: meetings inside long gaps (I and D breakpoints), rows that touch an end."""
    rng = np.random.default_rng(seed)

    def seq(n):
        return bytes(rng.choice(list(b"ACGT"), n).astype(np.uint8))

    pairs = [(seq(600), seq(600)), (seq(2200), seq(1300)), (seq(1200), seq(1900))]
    for n in range(700, 2400, 170):
        p = seq(n)
        t = _mutated(rng, p, n // 10, 3)
        gap, at = int(rng.integers(60, 300)), len(t) // 2 + int(rng.integers(-40, 40))
        pairs += [(p, t), (p, t[:at] + seq(gap) + t[at:]), (p, t[:at] + t[at + gap:])]
    b = pkg.PairBatch.from_lists([p for p, _ in pairs], [t for _, t in pairs])
    try:
        batch_aligner.set_exec_shape(gw, False)
        res = batch_aligner.align(b, penalties=pen)
    finally:
        batch_aligner.set_exec_shape(1, False)
    assert (res.status == 0).all()
    for i in range(b.n):
        _, score, ops, _ = binding.oracle_align(b.pattern(i), b.text(i), pen)
        assert res.scores[i] == score and pkg.runs_to_ops(res.runs_of(i)) == ops, (i, b.plen[i], b.tlen[i])


def test_small_batch_of_wide_pairs(batch_aligner):
    """A batch with a block for each pair starts in rings of full width: no pair is aligned twice, and
    the results are those of the first pass's capped rings with their retry pass."""
    rng = np.random.default_rng(31)

    def seq(n):
        return bytes(rng.choice(list(b"ACGT"), n).astype(np.uint8))

    p = seq(4000)
    pairs = [(seq(6000), seq(6000)), (p, _mutated(rng, p, 700, 3)), (seq(5000), b"A"), (seq(40), seq(50))]
    b = pkg.PairBatch.from_lists([p for p, _ in pairs], [t for _, t in pairs])
    res = batch_aligner.align(b)
    assert batch_aligner.stats().retried_pairs == 0
    capped = batch_aligner.align(b, sched=_capi.SCHED_PLAIN)
    assert batch_aligner.stats().retried_pairs > 0
    for i in range(b.n):
        _, score, ops, _ = binding.oracle_align(b.pattern(i), b.text(i))
        assert res.status[i] == capped.status[i] == 0 and res.scores[i] == capped.scores[i] == score, i
        assert pkg.runs_to_ops(res.runs_of(i)) == ops == pkg.runs_to_ops(capped.runs_of(i)), i
