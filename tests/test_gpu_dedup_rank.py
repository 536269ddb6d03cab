"""The simulated training set's dedup by one key per instance (the track's rank)
against the dedup of the same instances word by word: equal in every number.
Sizes on both sides of what one key holds."""
import numpy as np
import pytest

from whatprot_gb300.simulate import paper_model, random_dye_seqs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,C,most,P,per", [
    (16, 3, 5, 300, 20),
    (1, 1, 1, 7, 9),
    (5, 4, 3, 50, 11),
    (16, 4, 9, 60, 15),   # rank and id fill 64 bits or pass them: word by word
    (20, 2, 15, 40, 25),
    (16, 1, 15, 30, 33),
])
def test_ranked_dedup_matches_words(gpu_ctx, T, C, most, P, per):
    ds = random_dye_seqs(P, C, 6, 40, max_per_channel=most, min_total=1, seed=T + C)
    gpu_ctx.upload_model(paper_model(C), T)
    gpu_ctx.upload_peptides(ds)
    got, tracks, pep = gpu_ctx.simulate_dye_track_set(per, seed=3, instances=True)
    keep = tracks.reshape(len(tracks), -1).any(axis=1)
    ref = gpu_ctx.dedup_dye_tracks(tracks[keep].astype(np.int16).reshape(-1, T, C), ds.ids[pep[keep]],
                                   ds.counts[pep[keep]])
    for name in ("tracks", "src_off", "src_id", "src_count", "src_hits"):
        assert np.array_equal(getattr(got, name), getattr(ref, name)), name
