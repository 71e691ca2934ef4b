"""Tiles that a thread block's idle warps take (csrc/biwfa_tile_kernel.cuh) against the oracle, bit for
bit: several owners per block with jobs open at once, pairs of very different width beside each other,
one owner with all other warps helping."""
import ctypes as C

import numpy as np
import pytest

import biwfa_gpu_pii2025_gb300 as pkg
from oracle import binding

pytestmark = pytest.mark.gpu


def _pairs(rng, n):
    """Every eighth pair is wide (unrelated sequences of 300 - 1,200 bases), the others narrow or empty."""
    pairs = []
    for i in range(n):
        if i % 8 == 0:
            a, b = (rng.choice(list(b"ACGT"), int(rng.integers(300, 1200))).astype(np.uint8) for _ in range(2))
        else:
            a = rng.choice(list(b"ACGT"), int(rng.integers(0, 700))).astype(np.uint8)
            b = a.copy()
            for at in rng.integers(0, max(1, a.size), a.size // 25):
                b[at] = rng.choice(list(b"ACGT"))
            b = np.delete(b, rng.integers(0, a.size, a.size // 40)) if a.size else b
        pairs.append((bytes(a), bytes(b)))
    return pairs


@pytest.mark.parametrize("n,gw,seed", [(3, 1, 1), (200, 1, 2), (700, 1, 3), (400, 4, 4), (170, 8, 5)])
@pytest.mark.parametrize("metric,pen", [(binding.METRIC_AFFINE, (0, 4, 6, 2)), (binding.METRIC_LINEAR, (0, 4, 2, 0))])
def test_several_owners_share_helpers(batch_aligner, n, gw, seed, metric, pen):
    pairs = _pairs(np.random.default_rng(seed), n)
    b = pkg.PairBatch.from_lists([p for p, _ in pairs], [t for _, t in pairs])
    try:
        batch_aligner.set_exec_shape(gw, False)
        res = [batch_aligner.align(b, penalties=pen, metric=metric) for _ in range(2)]
    finally:
        batch_aligner.set_exec_shape(1, False)
    for r in res:
        assert (r.status == 0).all()
    for i in range(n):
        _, score, ops, _ = binding.oracle_align(b.pattern(i), b.text(i), pen, metric=metric)
        for r in res:
            assert pkg.runs_to_ops(r.runs_of(i)) == ops and r.scores[i] == (score if ops else 0), i


@pytest.mark.parametrize("n,lo,hi", [(20000, 1, 101), (3000, 101, 160)])
def test_every_root_is_aligned(batch_aligner, n, lo, hi):
    """The recursion's root is no stack entry: each pair, whether its root is a leaf (both sides up to
    100 bases) or a search, ends with the oracle's CIGAR and none with an empty one."""
    rng = np.random.default_rng(n)
    pairs = []
    for _ in range(n):
        p = rng.choice(list(b"ACGT"), int(rng.integers(lo, hi))).astype(np.uint8)
        t = p.copy()
        t[rng.integers(0, t.size)] = ord("C")
        pairs.append((bytes(p), bytes(np.append(t, t[:int(rng.integers(0, 4))]))))
    b = pkg.PairBatch.from_lists([p for p, _ in pairs], [t for _, t in pairs])
    res = batch_aligner.align(b)
    assert (res.status == 0).all() and (res.run_len > 0).all()
    for i in range(n):
        _, score, ops, _ = binding.oracle_align(b.pattern(i), b.text(i))
        assert pkg.runs_to_ops(res.runs_of(i)) == ops and res.scores[i] == score, i


@pytest.mark.parametrize("pen,seed", [((0, 31, 31, 0), 41), ((0, 28, 28, 0), 42), ((0, 7, 28, 0), 43), ((0, 31, 31, 0), 44)])
def test_widest_score_spacings(batch_aligner, pen, seed):
    """Gap-linear scores that hold a row lie up to 31 apart, the most that the score scope allows."""
    pairs = _pairs(np.random.default_rng(seed), 60)
    b = pkg.PairBatch.from_lists([p for p, _ in pairs], [t for _, t in pairs])
    res = batch_aligner.align(b, penalties=pen, metric=binding.METRIC_LINEAR)
    assert (res.status == 0).all()
    for i in range(b.n):
        _, score, ops, _ = binding.oracle_align(b.pattern(i), b.text(i), pen, metric=binding.METRIC_LINEAR)
        assert pkg.runs_to_ops(res.runs_of(i)) == ops and res.scores[i] == (score if ops else 0), i


def test_a_wait_that_runs_out_fails_the_run_and_leaves_the_context_usable(batch_aligner):
    """With one poll before a wait for a helper's tile has run out, the run ends with a device error and
    not with an alignment status; the next run, with the usual limit, is right."""
    rng = np.random.default_rng(51)
    pairs = [tuple(bytes(rng.choice(list(b"ACGT"), 3000).astype(np.uint8)) for _ in range(2)) for _ in range(4)]
    b = pkg.PairBatch.from_lists([p for p, _ in pairs], [t for _, t in pairs])
    limit = batch_aligner.lib.wfg_test_limit_waits
    limit.argtypes = [C.c_void_p, C.c_int]
    batch_aligner.upload(b)
    try:
        assert limit(batch_aligner.ctx, 1) == 0
        batch_aligner.run()
        with pytest.raises(RuntimeError, match="waited in vain"):
            batch_aligner.fetch()
        with pytest.raises(RuntimeError, match="waited in vain"):
            batch_aligner.synchronize()
    finally:
        assert limit(batch_aligner.ctx, 0) == 0
    res = batch_aligner.align(b)
    for i in range(b.n):
        _, score, ops, _ = binding.oracle_align(b.pattern(i), b.text(i))
        assert res.status[i] == 0 and res.scores[i] == score and pkg.runs_to_ops(res.runs_of(i)) == ops, i


@pytest.mark.parametrize("n", [152, 153, 320, 620])
def test_long_pairs_several_to_a_block(batch_aligner, n):
    """Pairs that start in rings of full width, as many as thread blocks, one more, two and up to four a
    block: low-error ones and some with wide wavefronts beside them."""
    rng = np.random.default_rng(n)
    pairs = []
    for i in range(n):
        p = rng.choice(list(b"ACGT"), int(rng.integers(16900, 17300))).astype(np.uint8)
        t = np.delete(p, rng.integers(0, p.size, 400 if i % 40 == 0 else 12))
        t[rng.integers(0, t.size, 8)] = ord("G")
        pairs.append((bytes(p), bytes(t)))
    b = pkg.PairBatch.from_lists([p for p, _ in pairs], [t for _, t in pairs])
    res = batch_aligner.align(b)
    assert batch_aligner.stats().retried_pairs == 0 and (res.status == 0).all()
    for i in range(n):
        _, score, ops, _ = binding.oracle_align(b.pattern(i), b.text(i))
        assert res.scores[i] == score and pkg.runs_to_ops(res.runs_of(i)) == ops, i
