"""The k-hit sets by levels where many tracks lie within the FP32 error of one
another's distance: k in the tens of thousands and more of half a million tracks, so
that groups of levels have to be taken in FP64 order and bins hold thousands of
tracks.  As test_gpu_khits.py: equal to the replayed search (the same set with a
fourth channel that shows no dyes, for interactions that act through it alone), and
found by levels, not left to that search."""
import numpy as np
import pytest

from whatprot_gb300.io import DyeTrackSet
from whatprot_gb300.simulate import paper_model, random_dye_seqs

pytestmark = pytest.mark.gpu


def test_dense(gpu_ctx):
    T, C, R = 16, 3, 150
    ds = random_dye_seqs(20000, C, 8, 40, max_per_channel=5, min_total=1, seed=1)
    gpu_ctx.upload_model(paper_model(C), T)
    gpu_ctx.upload_peptides(ds)
    dts = gpu_ctx.simulate_dye_track_set(60, seed=4321)
    reads, pep, _ = gpu_ctx.simulate_reads(R, seed=5)
    tracks = np.concatenate([dts.tracks, np.zeros((len(dts.tracks), T, 1), np.int16)], axis=2)
    dts = DyeTrackSet(tracks, dts.src_off, dts.src_id, dts.src_count, dts.src_hits)
    reads = np.concatenate([reads, np.zeros((R, T, 1))], axis=2)
    got = []
    for interacting in (False, True):
        sm = paper_model(C + 1)
        if interacting:
            sm.channel_models[0].flat_interactions[C] = 0.5
        gpu_ctx.upload_model(sm, T)
        gpu_ctx.upload_tracks(dts)
        gpu_ctx.set_nn_selection("kdtree")
        for k in (100000, 200000):
            got.append(gpu_ctx.nn_classify(reads, k, 0.5, 64))
            assert gpu_ctx.last_routes()["replayed"] == (R if interacting else 0)
    for a, b in ((got[0], got[2]), (got[1], got[3])):
        (n0, id0, sc0, tot0), (n1, id1, sc1, tot1) = a, b
        assert np.array_equal(n0, n1)
        assert np.allclose(tot0, tot1, rtol=1e-12, atol=0)
        assert np.allclose(sc0, sc1, rtol=1e-12, atol=0)
        for r in range(R):
            # ids of scores that differ by more than the rounding
            x = sc0[r, :n0[r]]
            b2 = np.concatenate([[-1.0], x, [np.inf]])
            alone = (x - b2[:-2] > 1e-10 * x) & (b2[2:] - x > 1e-10 * x)
            alone[0] = alone[0] and n0[r] < 64
            assert np.array_equal(id0[r, :n0[r]][alone], id1[r, :n0[r]][alone]), r


def test_distances_apart_in_64_bits_only(gpu_ctx):
    """Reads a hair (1e-9) from equal distances to whole families of tracks: the order
    within a family shows in the last bits of FP64, below FP32 and below the 32-bit keys
    that entries are ranked by first."""
    T, C, N, R, k = 6, 3, 5000, 60, 900
    rng = np.random.default_rng(12)
    tracks = rng.integers(0, 3, (2 * N, T, C)).astype(np.int16)
    tracks[:, :, C - 1] = 0
    tracks = np.unique(tracks.reshape(2 * N, -1), axis=0)
    tracks = tracks[rng.permutation(len(tracks))[:N]].reshape(-1, T, C)
    hits = np.minimum(rng.pareto(0.9, N) + 1, 50).astype(np.int32)
    dts = DyeTrackSet(tracks, np.arange(N + 1, dtype=np.int32), rng.integers(0, N // 4, N).astype(np.int32),
                      np.ones(N, np.int32), hits)
    reads = 1.3 + 0.3 * rng.integers(0, 2, (R, 1, 1)) + rng.random((R, T, C)) * 1e-9
    got = []
    for interacting in (False, True):
        sm = paper_model(C)
        if interacting:
            sm.channel_models[0].flat_interactions[C - 1] = 0.5
        gpu_ctx.upload_model(sm, T)
        gpu_ctx.upload_tracks(dts)
        gpu_ctx.set_nn_selection("kdtree")
        got.append(gpu_ctx.nn_classify(reads, k, 0.5, 64))
        if not interacting:
            assert gpu_ctx.last_routes()["levels"] >= R // 2
    (n0, id0, sc0, tot0), (n1, id1, sc1, tot1) = got
    assert np.array_equal(n0, n1)
    assert np.allclose(tot0, tot1, rtol=1e-12, atol=0)
    assert np.allclose(sc0, sc1, rtol=1e-12, atol=0)
