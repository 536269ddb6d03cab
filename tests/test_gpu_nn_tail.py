"""Places of a read's candidate list past its candidates: id 0, score 0, whatever
the memory held before (a call with more candidates), in both vote kernels and with
both selections."""
import numpy as np
import pytest

from whatprot_gb300.io import DyeTrackSet
from whatprot_gb300.simulate import paper_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("selection", ["kdtree", "prefix"])
@pytest.mark.parametrize("ids", [30, 40000])
def test_places_past_the_candidates(gpu_ctx, selection, ids):
    T, C, num, h = 6, 2, 400, 60
    rng = np.random.default_rng(3)
    t = np.maximum(rng.integers(0, 6, (num, 1, C)) - np.cumsum(rng.random((num, T, C)) < 0.3, axis=1), 0)
    t = np.unique(t.reshape(num, -1), axis=0).astype(np.int16).reshape(-1, T, C)
    S = max(len(t), ids)
    off = np.arange(len(t) + 1, dtype=np.int32)
    off[-1] = S
    dts = DyeTrackSet(t, off, (np.arange(S) % ids).astype(np.int32), np.ones(S, np.int32), np.ones(S, np.int32))
    reads = t[rng.integers(0, len(t) - 1, 50)] + rng.normal(0, 0.2, (50, T, C))
    gpu_ctx.upload_model(paper_model(C), T)
    gpu_ctx.set_nn_selection(selection)
    try:
        gpu_ctx.upload_tracks(dts)
        gpu_ctx.nn_classify(reads, 200, 0.5, h)
        for k in (5, 20):
            n, cid, sc, _ = gpu_ctx.nn_classify(reads, k, 0.5, h)
            assert n.min() < h
            for r in range(len(reads)):
                assert np.all(cid[r, :n[r]] >= 0) and np.all(sc[r, :n[r]] > 0), r
                assert np.all(cid[r, n[r]:] == 0) and np.all(sc[r, n[r]:] == 0), r
    finally:
        gpu_ctx.set_nn_selection("kdtree")
