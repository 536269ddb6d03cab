"""kNN against a large training set where the device has little memory left: the
level kernel's scratch (4.6 GB for 2,000 reads at k = 10,000) shrinks to what there
is, with the same results."""
import numpy as np
import pytest

from whatprot_gb300 import capi
from whatprot_gb300.simulate import paper_model, random_dye_seqs

pytestmark = pytest.mark.gpu


def test_little_memory_left(gpu_ctx):
    import torch
    T, C, R, k = 16, 3, 2000, 10000
    ds = random_dye_seqs(20000, C, 8, 40, max_per_channel=5, min_total=1, seed=1)
    ctx = capi.Context(0)
    try:
        ctx.upload_model(paper_model(C), T)
        ctx.upload_peptides(ds)
        ctx.simulate_dye_track_set(60, seed=4321, to_nn=True, download=False)
        reads, _, _ = ctx.simulate_reads(R, seed=5)
        ctx.nn_classify(reads[:2], k, 0.5, 20)  # the set's tables
        free = torch.cuda.mem_get_info()[0]
        hold = [torch.empty(free - (2 << 30), dtype=torch.uint8, device="cuda")]
        try:
            got = ctx.nn_classify(reads, k, 0.5, 20)
            routes = ctx.last_routes()
        finally:
            hold.clear()
            torch.cuda.empty_cache()
        want = ctx.nn_classify(reads, k, 0.5, 20)
        assert routes == ctx.last_routes()
        for x, y in zip(got, want):
            assert np.array_equal(x, y)
    finally:
        ctx.close()
