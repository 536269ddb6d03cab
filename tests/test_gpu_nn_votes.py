"""kNN votes (wp_nnscore.cu, and wp_nn.cu's select kernel beyond the ids that
shared memory holds) against the oracle, at the sizes where they change shape:
fewer ids than h, h of 1 and 1,024, a track with thousands of sources (several
slabs of pairs), kept sets around a multiple of 512, id counts on both sides of
what shared memory holds.

Scores are FP64 sums of positive terms; near weights are the oracle's own FP64
values, far ones FP32 (below 1e-8 of the largest weight): lists must match up to
ties at the h-th place, scores within 1e-5 of the list's largest, totals within
1e-5 (the tolerances of test_gpu_nn.py)."""
import numpy as np
import pytest

from conftest import nn_lists_match
from whatprot_gb300.io import DyeTrackSet
from whatprot_gb300.simulate import paper_model

pytestmark = pytest.mark.gpu

CASES = [
    # tracks, ids, sources of track 0, k, h
    (300, 3, 2, 60, 20),
    (700, 400, 5000, 512, 1),
    (1500, 5000, 9, 513, 1024),
    (2500, 20000, 3000, 900, 200),
    (3000, 40000, 9, 1100, 300),     # beyond shared memory
]


@pytest.mark.parametrize("selection", ["kdtree", "prefix"])
@pytest.mark.parametrize("case", CASES, ids=[f"n{c[0]}u{c[1]}s{c[2]}k{c[3]}h{c[4]}" for c in CASES])
def test_votes(gpu_ctx, oracle, case, selection):
    num, ids, first, k, h = case
    T, C = 8, 2
    rng = np.random.default_rng(num + ids)
    t = np.maximum(rng.integers(0, 8, (num, 1, C)) - np.cumsum(rng.random((num, T, C)) < 0.3, axis=1), 0)
    t = np.unique(t.reshape(num, -1), axis=0).astype(np.int16)
    t = t[rng.permutation(len(t))].reshape(-1, T, C)
    N = len(t)
    per = rng.integers(1, 4, N)
    per[0] = first
    per[-1] = max(per[-1], ids // N + 1)
    off = np.concatenate([[0], np.cumsum(per)]).astype(np.int32)
    S = int(off[-1])
    src = rng.integers(0, ids, S).astype(np.int32)
    src[rng.permutation(S)[:min(S, ids)]] = np.arange(min(S, ids), dtype=np.int32)
    if S < ids:  # the ids that no draw reached
        extra = np.arange(S, ids, dtype=np.int32)
        src, off[-1] = np.concatenate([src, extra]), off[-1] + len(extra)
        S = ids
    dts = DyeTrackSet(t, off, src, rng.integers(1, 4, S).astype(np.int32), rng.integers(1, 5, S).astype(np.int32))
    sm = paper_model(C)
    reads = t[rng.integers(0, N, 40)] + rng.normal(0, 0.25, (40, T, C))
    reads[0] = t[0] + 0.01
    gpu_ctx.upload_model(sm, T)
    gpu_ctx.upload_tracks(dts)
    gpu_ctx.set_nn_selection(selection)
    try:
        gn, gid, gsc, gtot = gpu_ctx.nn_classify(reads, k, 0.5, h)
    finally:
        gpu_ctx.set_nn_selection("kdtree")
    on, oid, osc, otot = oracle.nn_classify(sm, T, dts, reads, k, 0.5, h, selection=selection)
    for r in range(len(reads)):
        ok, _ = nn_lists_match(gid[r], gsc[r], gn[r], oid[r], osc[r], on[r], 1e-5)
        assert ok, r
        assert abs(gtot[r] - otot[r]) <= 1e-5 * otot[r], r
