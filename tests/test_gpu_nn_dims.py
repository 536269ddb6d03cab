"""The distance passes (two queries per lane) at the sizes where they change
shape: numbers of coordinates on both sides of each variant, entry counts that
end inside a tile or a super-tile and odd ones, read counts around a warp and a
CTA.  Prefix selection against the oracle, at the tolerance of test_gpu_nn.py for
that selection (2e-5: its boundary is decided in FP32)."""
import numpy as np
import pytest

from conftest import nn_lists_match
from whatprot_gb300.io import DyeTrackSet
from whatprot_gb300.simulate import paper_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,C,num,R", [
    (4, 1, 1, 1), (8, 1, 33, 33), (3, 3, 700, 31), (16, 1, 1025, 40), (12, 2, 2077, 65), (5, 4, 900, 64),
    (13, 2, 1500, 257), (16, 2, 63, 20), (12, 3, 3001, 300), (13, 3, 999, 17), (16, 3, 1057, 32), (14, 4, 555, 50),
    (15, 4, 1100, 16), (16, 4, 2049, 35),
])
def test_prefix_by_dimension(gpu_ctx, oracle, T, C, num, R):
    rng = np.random.default_rng(T * 100 + C * 10 + num)
    t = np.maximum(rng.integers(0, 7, (num, 1, C)) - np.cumsum(rng.random((num, T, C)) < 0.25, axis=1), 0)
    t = np.unique(t.reshape(num, -1), axis=0).astype(np.int16)
    t = t[rng.permutation(len(t))].reshape(-1, T, C)
    N = len(t)
    per = rng.integers(1, 4, N)
    off = np.concatenate([[0], np.cumsum(per)]).astype(np.int32)
    S = int(off[-1])
    dts = DyeTrackSet(t, off, rng.integers(0, max(2, N // 3), S).astype(np.int32),
                      rng.integers(1, 4, S).astype(np.int32), rng.integers(1, 6, S).astype(np.int32))
    sm = paper_model(C)
    reads = t[rng.integers(0, N, R)] + rng.normal(0, 0.3, (R, T, C))
    k, h = max(1, int(dts.src_hits.sum()) // 9), 25
    gpu_ctx.upload_model(sm, T)
    gpu_ctx.upload_tracks(dts)
    gpu_ctx.set_nn_selection("prefix")
    try:
        gn, gid, gsc, gtot = gpu_ctx.nn_classify(reads, k, 0.5, h)
    finally:
        gpu_ctx.set_nn_selection("kdtree")
    on, oid, osc, otot = oracle.nn_classify(sm, T, dts, reads, k, 0.5, h, selection="prefix")
    for r in range(R):
        ok, _ = nn_lists_match(gid[r], gsc[r], gn[r], oid[r], osc[r], on[r], 2e-5)
        assert ok, r
        assert abs(gtot[r] - otot[r]) <= 2e-5 * otot[r], r
