"""What a user of the aligner has it do, as cases that can be timed.

A batch case is one end-to-end call (BatchAligner.align_into): the pairs and the results lie in
page-locked host arrays, the call copies the pairs to the GPU, aligns them and copies scores,
statuses and CIGAR runs back. A "one" case is one call of the WFA2-lib style single-pair API. The
"train" case trains the schedule's score predictor on a resident batch.

Cases, their fields and what they stand for:
  path     "batch", "one" or "train"
  pairs    pairs in the batch
  lo, hi   pattern lengths, log-uniform in [lo, hi]; mix: thirds of 1,000 bp, 150 bp and [lo, hi]
  err_lo, err_hi  edit events per base, per pair uniform (a third each of substitutions,
           insertions and deletions; gap lengths geometric with mean `gap`)
  with_n   share of pairs that hold some N bases (compared as bytes, not as 2-bit codes)
  metric, pen  distance and penalties (match, mismatch, gap opening, gap extension, ...)
  score_only, learned  options of the call
"""
import math

import numpy as np
import torch

import biwfa_gpu_pii2025_gb300 as pkg
from biwfa_gpu_pii2025_gb300 import _capi

METRICS = {"affine": _capi.METRIC_GAP_AFFINE, "edit": _capi.METRIC_EDIT, "indel": _capi.METRIC_INDEL,
           "linear": _capi.METRIC_GAP_LINEAR, "affine2p": _capi.METRIC_GAP_AFFINE_2P}
AFFINE = "0,4,6,2"           # WFA2-lib's defaults, the penalties of every benchmark workload here
AFFINE2P = "0,4,6,2,24,1"    # WFA2-lib's two-piece defaults


def _case(name=None, path="batch", pairs=1, lo=1000, hi=1000, err_lo=0.05, err_hi=0.05, gap=1, with_n=0.0, mix=False,
          metric="affine", pen=AFFINE, score_only=False, learned=False):
    c = dict(path=path, pairs=pairs, lo=lo, hi=hi, err_lo=err_lo, err_hi=err_hi, gap=gap, with_n=with_n, mix=mix,
             metric=metric, pen=pen, score_only=score_only, learned=learned)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # One short read through wavefront_align(): the smallest call, all latency.
        _case("one_150bp", path="one", lo=150, hi=150, err_lo=0.02, err_hi=0.02),
        # One long pair through wavefront_align(): an interactive call on a gene-sized sequence.
        _case("one_10kbp", path="one", lo=10000, hi=10000, err_lo=0.05, err_hi=0.05, gap=2),
        # A small batch of 1 kbp pairs, far fewer than the GPU holds at once.
        _case("kbp_64", pairs=64),
        # The 1 kbp / 5 % workload of the benchmark.
        _case("kbp_10k", pairs=10000),
        # Short reads, some with N bases, as a sequencer delivers them.
        _case("reads_200k", pairs=200000, lo=150, hi=150, err_lo=0.02, err_hi=0.02, with_n=0.02),
        # The uneven workload of the benchmark: 100 bp to 10 kbp, 1-10 % error.
        _case("uneven_20k", pairs=20000, lo=100, hi=10000, err_lo=0.01, err_hi=0.10, gap=2),
        # The benchmark's mixture on the learned schedule, input copies overlapped with the alignment.
        _case("mixture_150k", pairs=150000, lo=100, hi=10000, err_lo=0.01, err_hi=0.10, gap=2, mix=True, learned=True),
        # Long noisy reads: wide wavefronts, deep recursion.
        _case("noisy_long_48", pairs=48, lo=10000, hi=20000, err_lo=0.12, err_hi=0.12, gap=2),
        # Scores only, as a filter that ranks candidates asks for them.
        _case("score_only_10k", pairs=10000, lo=200, hi=5000, err_lo=0.01, err_hi=0.10, gap=2, score_only=True),
        # Edit distance over uneven pairs.
        _case("edit_20k", pairs=20000, lo=100, hi=10000, err_lo=0.01, err_hi=0.10, metric="edit", pen="0,1,0,0"),
        # Two-piece gap-affine, the long-read distance.
        _case("affine2p_4k", pairs=4000, lo=100, hi=3000, err_lo=0.01, err_hi=0.08, gap=2, metric="affine2p",
              pen=AFFINE2P),
        # Training of the learned schedule's predictor on scored pairs.
        _case("train_16k", path="train", pairs=16384, lo=100, hi=2000, err_lo=0.01, err_hi=0.10, gap=2),
    ]


# Relative cost of a distance's alignment against the default gap-affine one.
_WEIGHT = {"affine": 1.0, "edit": 0.3, "indel": 0.3, "linear": 0.5, "affine2p": 12.0}
_PENALTIES = {"affine": [AFFINE, AFFINE, AFFINE, "0,4,6,1", "0,2,3,1", "-1,4,6,2", "0,5,8,2"], "edit": ["0,1,0,0"],
              "indel": ["0,1,0,0"], "linear": ["0,4,2", "0,4,6"], "affine2p": [AFFINE2P]}


def _spread(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    path = rng.choice(["batch"] * 8 + ["one", "train"])
    if path == "train":
        return _case(path="train", pairs=int(_spread(rng, 1000, 16384)), lo=100, hi=rng.randint(200, 2000), err_lo=0.01,
                     err_hi=round(rng.uniform(0.02, 0.10), 3), gap=2)
    metric = rng.choice(["affine"] * 6 + ["edit", "indel", "linear", "affine2p"])
    hi = int(_spread(rng, 60, 12000))
    lo = hi if path == "one" else max(40, int(hi / _spread(rng, 1, 60)))
    gap = rng.choice([1, 2, 3])
    err_hi = round(_spread(rng, 0.01, 0.12), 3)
    # An estimate of the call's time: a pair's work grows with the square of its edits.
    edits = err_hi * hi * (1 + 0.5 * (gap - 1)) * math.sqrt(_WEIGHT[metric])
    while edits > 800:  # the longest single pair
        hi, lo = max(60, int(hi * 0.7)), max(40, int(lo * 0.7))
        edits = err_hi * hi * (1 + 0.5 * (gap - 1)) * math.sqrt(_WEIGHT[metric])
    lo = min(lo, hi)
    pairs = 1 if path == "one" else int(_spread(rng, 3, min(150000, 0.15 / (1.7e-10 * edits * edits + 1e-7), 6e7 / hi)))
    return _case(path=path, pairs=max(1, pairs), lo=lo, hi=hi, err_lo=round(err_hi * rng.uniform(0.2, 1), 4),
                 err_hi=err_hi, gap=gap, with_n=rng.choice([0.0, 0.0, 0.05]), metric=metric,
                 pen=rng.choice(_PENALTIES[metric]), score_only=path == "batch" and rng.random() < 0.15)


def _pairs(case, seed):
    """Pairs of the case's shape, made on the GPU: ASCII bytes, offsets and lengths on the host."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def rand(n):
        return torch.rand(n, generator=g, device="cuda")

    def ints(n, top):
        return torch.randint(0, top, (n,), generator=g, device="cuda", dtype=torch.uint8)

    n, lo, hi = case["pairs"], case["lo"], case["hi"]
    u = rand(n).double()
    plen = torch.exp(math.log(lo) + u * (math.log(hi + 1) - math.log(lo))).long().clamp(lo, hi)
    err = case["err_lo"] + rand(n) * (case["err_hi"] - case["err_lo"])
    gap = torch.full((n,), float(case["gap"]), device="cuda")
    if case["mix"]:
        kind = ints(n, 3)
        plen = torch.where(kind == 0, 1000, torch.where(kind == 1, 150, plen))
        err = torch.where(kind == 0, 0.05, torch.where(kind == 1, 0.02, err))
        gap = torch.where(kind == 2, gap, 1.0)
    total = int(plen.sum())
    end = plen.cumsum(0)
    of = torch.repeat_interleave(torch.arange(n, device="cuda", dtype=torch.int32), plen)
    code = ints(total, 4)
    if case["with_n"] > 0:
        code[(rand(n) < case["with_n"])[of.long()] & (rand(total) < 0.01)] = 4
    event = rand(total) < err[of.long()]
    kind = ints(total, 3)
    # geometric lengths with mean `gap`: 1 + floor(log u / log(1 - 1/gap))
    p = 1.0 - 1.0 / gap[of.long()]
    length = torch.where(p > 0, 1 + torch.floor(torch.log(rand(total).clamp_min(1e-6)) / torch.log(p.clamp_min(1e-6))), 1.0)
    length = length.clamp(1, 60).int()
    at = torch.nonzero(event & (kind == 2)).squeeze(1)
    cover = torch.zeros(total + 1, device="cuda", dtype=torch.int32)
    cover.index_add_(0, at, torch.ones_like(at, dtype=torch.int32))
    stop = torch.minimum(at + length[at], end[of[at].long()])
    cover.index_add_(0, stop, torch.full_like(at, -1, dtype=torch.int32))
    gone = cover.cumsum(0)[:total] > 0
    more = torch.where(event & (kind == 1), length, 0)
    count = more + (~gone).int()
    after = count.cumsum(0)
    sub = event & (kind == 0) & (code < 4)
    new = torch.where(sub, (code + 1 + ints(total, 3)) % 4, code)
    text = ints(int(after[-1]), 4)
    text[(after - 1)[~gone].long()] = new[~gone]
    tend = after[end - 1].long()
    tlen = torch.diff(tend, prepend=tend.new_zeros(1))
    table = torch.tensor([65, 67, 71, 84, 78], device="cuda", dtype=torch.uint8)
    seq = torch.cat([table[code.long()], table[text.long()]]).cpu().numpy()
    p_off, t_off = (end - plen).cpu().numpy(), (tend - tlen).cpu().numpy() + total
    return pkg.PairBatch(seq, p_off.astype(np.int64), plen.cpu().numpy().astype(np.int32), t_off.astype(np.int64),
                         tlen.cpu().numpy().astype(np.int32))


def _penalties(case):
    v = [int(x) for x in case["pen"].split(",")]
    return tuple(v + [0] * (4 - len(v)))


class _State:
    """The handles and buffers of one case; freed with it."""

    def __init__(self, case):
        self.case, self.penalties, self.metric = case, _penalties(case), METRICS[case["metric"]]
        self.opened = []

    def keep(self, handle):
        self.opened.append(handle)
        return handle

    def __del__(self):
        for h in reversed(self.opened):
            h.close()


def prepare(case, seed):
    s = _State(case)
    b = _pairs(case, seed)
    if case["path"] == "one":
        p = s.penalties
        distance = {"affine": _capi.GAP_AFFINE, "edit": _capi.EDIT, "indel": _capi.INDEL, "linear": _capi.GAP_LINEAR,
                    "affine2p": _capi.GAP_AFFINE_2P}[case["metric"]]
        two = dict(gap_opening2=p[4], gap_extension2=p[5]) if len(p) > 4 else {}
        s.aligner = s.keep(pkg.WavefrontAligner(*p[:4], distance=distance, **two))
        s.pattern, s.text = b.pattern(0), b.text(0)
        return s
    s.aligner = s.keep(pkg.BatchAligner(0))
    if case["path"] == "train":
        s.scores = s.aligner.align(b, score_only=True).scores
        s.model = s.keep(pkg.ScorePredictor(s.aligner, seed=1))
        s.start = _start_params(seed)
        return s
    if case["learned"]:
        sample = b.subset(range(0, b.n, max(1, b.n // 2048)))
        scores = s.aligner.align(sample, score_only=True).scores
        s.model = s.keep(pkg.ScorePredictor(s.aligner, seed=1))
        s.model.train(scores, epochs=20, batch_rows=256)
        s.model.attach()
        s.aligner.set_learned_policy(3.4e38, 8, False, 1.4)  # one warp per pair throughout
    pin = s.keep(pkg.PinnedHost())
    s.batch = pin.batch(b)
    n, runs = b.n, _most_runs(case)
    s.out = pkg.BatchResult(pin.empty(n, np.int32), pin.empty(n, np.int32), pin.empty(n, np.int64),
                            pin.empty(n, np.int32), pin.empty(runs, np.uint32))
    return s


def run(s):
    c = s.case
    if c["path"] == "one":
        status = s.aligner.align(s.pattern, s.text)
        ops = np.frombuffer(s.aligner.cigar_ops().encode(), np.uint8)
        return status, s.aligner.score, np.pad(ops, (0, 3 * c["hi"] + 64 - ops.size))
    if c["path"] == "train":
        s.model.set_params(s.start)
        losses = s.model.train(s.scores, epochs=2, batch_rows=2048, lr=2e-3, seed=7)
        return losses, s.model.params()
    sched = _capi.SCHED_LEARNED if c["learned"] else _capi.SCHED_SORTED
    total = s.aligner.align_into(s.batch, s.out, penalties=s.penalties, score_only=c["score_only"], sched=sched,
                                 metric=s.metric)
    # The results as tensors of their own (the page-locked arrays are written again by the next call).
    scores, status = torch.from_numpy(s.out.scores).cuda(), torch.from_numpy(s.out.status).cuda()
    if c["score_only"]:
        return scores, status
    # The runs of all pairs in the pairs' order (a pair's place in `runs` depends on when it finished).
    off, length = torch.from_numpy(s.out.run_off).cuda(), torch.from_numpy(s.out.run_len).cuda()
    shift = torch.repeat_interleave(off - (length.cumsum(0) - length), length.long(), output_size=total)
    runs = torch.zeros(_most_runs(c), device="cuda", dtype=torch.int32)
    runs[:total] = torch.from_numpy(s.out.runs[:total].view(np.int32)).cuda()[torch.arange(total, device="cuda") + shift]
    return scores, status, length, runs


def _mean_length(case):
    lo, hi = case["lo"], case["hi"]
    mean = (hi - lo) / math.log(hi / lo) if hi > lo else hi
    return (1000 + 150 + mean) / 3 if case["mix"] else mean


def _most_runs(case):
    """Room for the CIGAR runs of a batch: an edit ends at most two runs; few pairs may all be long ones."""
    edits = (_mean_length(case) if case["pairs"] >= 1000 else case["hi"]) * case["err_hi"]
    return int(case["pairs"] * (4 * edits + 24))


def work(case):
    if case["path"] == "train":
        # two epochs of forward (32 x 64 and 64 x 64 products) and the backward's two products of each
        macs = 2 * case["pairs"] * 3 * (32 * 64 + 64 * 64 + 64)
        return {"bytes": 2 * case["pairs"] * 32 * 2 + 3 * 4 * 6465, "flops": 2 * macs}
    mean = _mean_length(case)
    edits = mean * 0.5 * (case["err_lo"] + case["err_hi"])
    # both sequences in; score, status and the CIGAR's runs (about two an edit) out
    return {"bytes": case["pairs"] * (2 * mean + 8 + (0 if case["score_only"] else 8 * edits + 4)), "flops": 0}


# ---- the predictor in 64 bits (exact): features, network, mean squared error, Adam
_IN, _HID = 32, 64


def _start_params(seed):
    r = np.random.default_rng(seed)
    a1, a2 = math.sqrt(6 / _IN), math.sqrt(6 / _HID)
    return np.concatenate([r.uniform(-a1, a1, _IN * _HID), np.zeros(_HID), r.uniform(-a2, a2, _HID * _HID), np.zeros(_HID),
                           r.uniform(-a2, a2, _HID) * 0.5, np.zeros(1)]).astype(np.float32)


def _features(b):
    n = b.n

    def counts(off, length):
        c = np.zeros((n, 256))
        for i in range(n):
            a = (b.seq[off[i]:off[i] + length[i]] >> 1) & 3
            if a.size >= 4:
                c[i] = np.bincount((a[:-3] << 6) | (a[1:-2] << 4) | (a[2:-1] << 2) | a[3:], minlength=256)
        return c

    d = np.abs(counts(b.p_off, b.plen) - counts(b.t_off, b.tlen)).astype(np.int64)
    at = np.where(d < 16, d, np.minimum(27, 12 + np.floor(np.log2(np.maximum(d, 1))).astype(np.int64)))
    p, t = b.plen.astype(np.float64), b.tlen.astype(np.float64)
    hist = np.zeros((n, 28))
    np.add.at(hist, (np.repeat(np.arange(n), 256), at.reshape(-1)), 1)
    return np.concatenate([np.log2(p + 1)[:, None] / 16, np.log2(t + 1)[:, None] / 16, ((p - t) / (p + t + 1))[:, None],
                           hist / 256, (d.sum(1) / (p + t + 1))[:, None]], axis=1)


def _orders(n, epochs, seed):
    """The epochs' row orders: a Fisher-Yates shuffle driven by splitmix64, carried from epoch to epoch."""
    mask, x, rows = (1 << 64) - 1, seed, list(range(n))
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            x = (x + 0x9E3779B97F4A7C15) & mask
            z = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = ((z ^ (z >> 31)) * (i + 1)) >> 64
            rows[i], rows[j] = rows[j], rows[i]
        yield np.array(rows)


def exact(case, seed):
    if case["path"] != "train":
        return None  # scores, statuses and CIGARs are whole numbers
    s = prepare(case, seed)
    target = np.log1p(np.abs(s.scores.astype(np.float64)))
    x = _features(_pairs(case, seed))
    cut = np.cumsum([_IN * _HID, _HID, _HID * _HID, _HID, _HID])
    par = s.start.astype(np.float64)
    m, v, step, losses = np.zeros_like(par), np.zeros_like(par), 0, []
    for rows in _orders(case["pairs"], 2, 7):
        loss = 0.0
        for k in range(0, len(rows), 2048):
            at = rows[k:k + 2048]
            w1, b1, w2, b2, w3, b3 = np.split(par, cut)
            w1, w2 = w1.reshape(_IN, _HID), w2.reshape(_HID, _HID)
            h1 = np.maximum(x[at] @ w1 + b1, 0)
            h2 = np.maximum(h1 @ w2 + b2, 0)
            e = h2 @ w3 + b3 - target[at]
            loss += float((e * e).sum())
            dy = 2 * e / len(at)
            d2 = dy[:, None] * w3 * (h2 > 0)
            d1 = (d2 @ w2.T) * (h1 > 0)
            g = np.concatenate([(x[at].T @ d1).ravel(), d1.sum(0), (h1.T @ d2).ravel(), d2.sum(0), h2.T @ dy, [dy.sum()]])
            step += 1
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            par = par - 2e-3 * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        losses.append(loss / len(rows))
    return np.array(losses), par
