"""The k-hit sets found by levels (wp_khits.cu) against the replayed search
(wp_kbest.cu) on the GPU.

A model with dye interactions takes the replay; one whose interactions only
act through a channel that no track has dyes on has the same coordinates, so
the same tree and the same k-hit sets.  Both routes then weigh the same kept
tracks, so every output must be equal: candidate counts and ids exactly,
scores and totals to the rounding of FP64 sums of up to a few thousand
positive terms in two orders (1e-12)."""
import numpy as np
import pytest

from whatprot_gb300.io import DyeTrackSet
from whatprot_gb300.simulate import paper_model

pytestmark = pytest.mark.gpu


def _tracks(rng, N, T, C, most):
    """N dye-tracks (falling counts) whose last channel never shows a dye,
    skewed hits, one to three sources each."""
    start = rng.integers(0, most + 1, (N, 1, C))
    t = np.maximum(start - np.cumsum(rng.random((N, T, C)) < 0.25, axis=1), 0).astype(np.int16)
    t[:, :, C - 1] = 0
    t = np.unique(t.reshape(N, -1), axis=0)
    t = t[rng.permutation(len(t))].reshape(-1, T, C)
    per = rng.integers(1, 4, len(t))
    off = np.concatenate([[0], np.cumsum(per)]).astype(np.int32)
    S = int(off[-1])
    hits = np.minimum(rng.pareto(0.9, S) + 1, 300).astype(np.int32)
    return DyeTrackSet(t, off, rng.integers(0, max(2, len(t) // 4), S).astype(np.int32), np.ones(S, np.int32), hits)


CASES = [
    # T, C, most dyes, tracks drawn, k (-1: every hit), noise of the reads
    (8, 2, 5, 3000, 200, 0.3),
    (16, 3, 5, 6000, 1000, 0.3),    # DP 48, several leaves
    (16, 4, 15, 4000, 300, 0.4),    # DP 64, counts up to 15
    (5, 2, 3, 400, 1, 0.3),         # k = 1
    (12, 2, 6, 5000, 17, 0.3),      # small leaves
    (16, 3, 4, 129, 40, 0.3),       # one entry beyond a group of 128
    (9, 3, 5, 2500, -1, 0.3),       # k = all hits
    (8, 2, 4, 2000, 150, 0.0),      # whole-number reads: equal distances
    (16, 3, 5, 20000, 4000, 0.02),  # reads almost on a track
    (16, 3, 5, 40000, 15000, 0.4),  # many groups looked into, by several warps
    (4, 2, 15, 900, 60, 3.0),       # reads far from every track
]


@pytest.mark.parametrize("case", CASES, ids=[f"T{c[0]}C{c[1]}d{c[2]}n{c[3]}k{c[4]}s{c[5]}" for c in CASES])
def test_levels_equal_replay(gpu_ctx, case):
    T, C, most, num, k, noise = case
    rng = np.random.default_rng(1000 + num + T)
    dts = _tracks(rng, num, T, C, most)
    k = int(dts.src_hits.sum()) if k < 0 else k
    at = rng.integers(0, len(dts.tracks), 150)
    reads = dts.tracks[at].astype(np.float64)
    reads += rng.normal(0, noise, reads.shape) if noise else 0.0
    got = []
    for interacting in (False, True):
        sm = paper_model(C)
        if interacting:
            sm.channel_models[0].flat_interactions[C - 1] = 0.5
        gpu_ctx.upload_model(sm, T)
        gpu_ctx.upload_tracks(dts)
        gpu_ctx.set_nn_selection("kdtree")
        got.append(gpu_ctx.nn_classify(reads, k, 0.5, 64))
    (n0, id0, sc0, tot0), (n1, id1, sc1, tot1) = got
    assert np.array_equal(n0, n1)
    assert np.allclose(tot0, tot1, rtol=1e-12, atol=0)
    for r in range(len(n0)):
        assert np.allclose(sc0[r, :n0[r]], sc1[r, :n0[r]], rtol=1e-12, atol=0), r
        # ids of scores that differ by more than the rounding
        a, b = sc0[r, :n0[r]], np.concatenate([[-1.0], sc0[r, :n0[r]], [np.inf]])
        alone = (a - b[:-2] > 1e-10 * a) & (b[2:] - a > 1e-10 * a)
        alone[0] = alone[0] and n0[r] < 64
        assert np.array_equal(id0[r, :n0[r]][alone], id1[r, :n0[r]][alone]), r
