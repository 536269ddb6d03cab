"""kNN votes of reads that are not finite, or so large that FP32 distances overflow:
their scores are NaN, which no sort of the candidates may let push its padding into
the list.  Such reads name candidates of the training set, and the other reads of
the batch keep their results, bit for bit.  With the scores in shared memory and,
for large sets of ids, in global memory."""
import numpy as np
import pytest

from whatprot_gb300.io import DyeTrackSet
from whatprot_gb300.simulate import paper_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ids", [37, 40000])
@pytest.mark.parametrize("value", [np.nan, -np.nan, np.inf, -np.inf, 1e30])
def test_nonfinite_read(gpu_ctx, value, ids):
    T, C, num = 6, 2, 500
    rng = np.random.default_rng(7)
    t = np.maximum(rng.integers(0, 6, (num, 1, C)) - np.cumsum(rng.random((num, T, C)) < 0.3, axis=1), 0)
    t = np.unique(t.reshape(num, -1), axis=0).astype(np.int16).reshape(-1, T, C)
    S = max(len(t), ids)
    off = np.arange(len(t) + 1, dtype=np.int32)
    off[-1] = S
    dts = DyeTrackSet(t, off, (np.arange(S) % ids).astype(np.int32), np.ones(S, np.int32), np.ones(S, np.int32))
    reads = t[rng.integers(0, len(t), 40)] + rng.normal(0, 0.2, (40, T, C))
    bad = reads.copy()
    bad[11] = bad[30] = value
    if np.isfinite(value) or np.isinf(value):  # a NaN among numbers is refused (its distances fit no bin)
        bad[11] = reads[11]
        bad[11, 2, 1] = value
    gpu_ctx.upload_model(paper_model(C), T)
    gpu_ctx.upload_tracks(dts)
    gpu_ctx.set_nn_selection("prefix")
    try:
        for h in (5, 300):  # fewer and more than the ids voted for
            n, cid, sc, tot = gpu_ctx.nn_classify(reads, 60, 0.5, h)
            bn, bid, bsc, btot = gpu_ctx.nn_classify(bad, 60, 0.5, h)
            for r in range(len(reads)):
                if r in (11, 30):
                    assert np.all((bid[r, :bn[r]] >= 0) & (bid[r, :bn[r]] < ids)), r
                    continue
                assert n[r] == bn[r] and tot[r] == btot[r], r
                assert np.array_equal(cid[r, :n[r]], bid[r, :n[r]]), r
                assert np.array_equal(sc[r, :n[r]], bsc[r, :n[r]]), r
    finally:
        gpu_ctx.set_nn_selection("kdtree")
