"""Which route the calls took (wp_last_routes) that other tests compare two routes of:
a comparison of the replayed search with itself, or of word keys with word keys, would
pass whatever the other route does.  The cases are those tests' own."""
from math import comb

import numpy as np
import pytest

from test_gpu_dedup_rank import test_ranked_dedup_matches_words as ranked_dedup
from test_gpu_khits import CASES, _tracks
from whatprot_gb300.simulate import paper_model, random_dye_seqs

pytestmark = pytest.mark.gpu
DEDUP = next(m for m in ranked_dedup.pytestmark if m.name == "parametrize").args[1]


@pytest.mark.parametrize("case", CASES, ids=[f"T{c[0]}C{c[1]}d{c[2]}n{c[3]}k{c[4]}s{c[5]}" for c in CASES])
def test_levels_answer(gpu_ctx, case):
    T, C, most, num, k, noise = case
    rng = np.random.default_rng(1000 + num + T)
    dts = _tracks(rng, num, T, C, most)
    k = int(dts.src_hits.sum()) if k < 0 else k
    reads = dts.tracks[rng.integers(0, len(dts.tracks), 150)].astype(np.float64)
    reads += rng.normal(0, noise, reads.shape) if noise else 0.0
    sm = paper_model(C)
    for interacting in (False, True):
        if interacting:
            sm.channel_models[0].flat_interactions[C - 1] = 0.5
        gpu_ctx.upload_model(sm, T)
        gpu_ctx.upload_tracks(dts)
        gpu_ctx.set_nn_selection("kdtree")
        gpu_ctx.nn_classify(reads, k, 0.5, 64)
        got = gpu_ctx.last_routes()
        assert got["levels"] + got["replayed"] == 150
        if interacting:
            assert got["levels"] == 0
        elif k < 4:
            assert got["levels"] == 0  # leaves of a few tracks: the search as it is
        elif noise:
            assert got["replayed"] == 0
        else:
            assert got["replayed"] > 0  # whole-number reads: equal distances


@pytest.mark.parametrize("k,R,levels", [(1, 60, False), (2, 60, False), (3, 60, False), (4, 60, True), (4, 16, True),
                                        (4, 15, False), (23, 15, False), (24, 15, True), (24, 1, True), (23, 1, False)])
def test_least_k(gpu_ctx, k, R, levels):
    """The line between the search and the levels."""
    dts = _tracks(np.random.default_rng(8), 4000, 12, 3, 5)
    reads = dts.tracks[:R] + np.random.default_rng(9).normal(0, 0.3, (R, 12, 3))
    gpu_ctx.upload_model(paper_model(3), 12)
    gpu_ctx.upload_tracks(dts)
    gpu_ctx.nn_classify(reads, k, 0.5, 8)
    got = gpu_ctx.last_routes()
    assert (got["levels"], got["replayed"]) == ((R, 0) if levels else (0, R))


@pytest.mark.parametrize("T,C,most,P,per", DEDUP)
def test_dedup_keys(gpu_ctx, T, C, most, P, per):
    ds = random_dye_seqs(P, C, 6, 40, max_per_channel=most, min_total=1, seed=T + C)
    gpu_ctx.upload_model(paper_model(C), T)
    gpu_ctx.upload_peptides(ds)
    got, tracks, pep = gpu_ctx.simulate_dye_track_set(per, seed=3, instances=True)
    dyes = max(int((s == c).sum()) for s in ds.seqs for c in range(C))
    bits = (comb(T + dyes, dyes) ** C).bit_length() + int(ds.ids.max() - ds.ids.min()).bit_length()
    assert gpu_ctx.last_routes()["dedup"] == ("rank" if bits <= 64 else "words")
    gpu_ctx.dedup_dye_tracks(tracks[:5].astype(np.int16).reshape(-1, T, C), ds.ids[pep[:5]], ds.counts[pep[:5]])
    assert gpu_ctx.last_routes()["dedup"] == "words"


def test_dedup_cases_on_both_sides():
    sides = set()
    for T, C, most, P, _ in DEDUP:
        ds = random_dye_seqs(P, C, 6, 40, max_per_channel=most, min_total=1, seed=T + C)
        dyes = max(int((s == c).sum()) for s in ds.seqs for c in range(C))
        sides.add((comb(T + dyes, dyes) ** C).bit_length() + int(ds.ids.max() - ds.ids.min()).bit_length() <= 64)
    assert sides == {True, False}
