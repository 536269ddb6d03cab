"""Classify calls on both sides of the batch size up to which the outputs go
through page-locked memory: the same numbers as in one large batch, read by read
(the arithmetic of a read does not depend on its batch)."""
import numpy as np
import pytest

from whatprot_gb300.simulate import paper_model, random_dye_seqs, simulate_radiometries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 33, 4096, 4097])
def test_batch_sizes_agree(gpu_ctx, R):
    sm = paper_model(2)
    ds = random_dye_seqs(15, 2, 6, 16, max_per_channel=4, min_total=1, seed=3)
    rads, _ = simulate_radiometries(sm, ds, 8, 4600, seed=4)
    gpu_ctx.upload_model(sm, 8)
    gpu_ctx.upload_peptides(ds)
    whole = gpu_ctx.classify(rads, 5.0)
    part = gpu_ctx.classify(rads[:R], 5.0)
    for a, b in zip(part, whole):
        assert np.array_equal(a, b[:R])
