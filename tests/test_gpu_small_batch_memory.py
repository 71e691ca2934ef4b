"""Device memory that a small batch takes: arenas for its pairs, not for every warp of the GPU."""
import numpy as np
import pytest
import torch

import biwfa_gpu_pii2025_gb300 as pkg
from oracle import binding

pytestmark = pytest.mark.gpu


# An arena of the 1 kbp pairs is 1.5 MB in the first pass (two rings of 12 rows of three components and
# 4,096 diagonals, 256 KiB of leaf store) and 4.5 MB in the last retry pass (3.2 MB of leaf store); of the
# 10 kbp pairs 1.7 and 13 MB (rings of 32,768 diagonals), of the 150 bp pair 0.5 and 1.8 MB. The bound is
# the pairs, of which at most one a block of 152 in the retry passes, times the larger, plus 64 MB for
# the batch itself, its results and the allocator's blocks.
@pytest.mark.parametrize("n,length,bound_mb", [(1, 150, 66), (64, 1000, 64 * 4.5 + 64), (200, 10000, 152 * 13 + 64)])
def test_small_batch_reserves_arenas_for_its_pairs(n, length, bound_mb):
    rng = np.random.default_rng(n)
    pairs = []
    for _ in range(n):
        p = rng.choice(list(b"ACGT"), length).astype(np.uint8)
        t = p.copy()
        t[rng.integers(0, length, length // 100)] = ord("A")
        pairs.append((bytes(p), bytes(t)))
    b = pkg.PairBatch.from_lists([p for p, _ in pairs], [t for _, t in pairs])
    warm = pkg.BatchAligner(0)  # the library's code and the context's own buffers are on the device
    warm.align(pkg.PairBatch.from_lists([b"ACGT"], [b"ACGA"]))
    torch.cuda.init()
    before = torch.cuda.mem_get_info(0)[0]
    al = pkg.BatchAligner(0)
    res = al.align(b)
    used = before - torch.cuda.mem_get_info(0)[0]
    al.close()
    warm.close()
    assert used <= bound_mb * 1e6, used
    assert (res.status == 0).all()
    for i in range(0, n, max(1, n // 8)):
        _, score, ops, _ = binding.oracle_align(b.pattern(i), b.text(i))
        assert res.scores[i] == score and pkg.runs_to_ops(res.runs_of(i)) == ops
