"""The pair engine with several lanes per pair (pairs with large boxes)
against the engine with one thread per pair: the same arithmetic in the same
order, so the results have the same bits."""
import numpy as np
import pytest

from oracle_lib import DBL_MAX
from test_gpu_forward import _model, assert_logp_close
from whatprot_gb300.model import DyeSeqSet, parse_dye_seq
from whatprot_gb300.simulate import random_dye_seqs, simulate_radiometries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,T,maxc,cut,block,inter", [
    (3, 16, 3, DBL_MAX, False, False),   # narrow boxes, full size
    (3, 16, 5, DBL_MAX, False, False),   # boxes wider than 4 as well
    (3, 16, 5, 5.0, False, False),       # boxes that move and shrink
    (3, 11, 4, DBL_MAX, True, False),    # broken-N states
    (2, 12, 7, 3.0, True, False),
    (1, 17, 9, DBL_MAX, False, False),   # one channel, the last packed length
    (2, 20, 4, DBL_MAX, False, False),   # positions past the packed codes
    (4, 8, 2, DBL_MAX, False, False),
    (4, 7, 3, 5.0, True, False),
    (3, 9, 3, DBL_MAX, False, True),     # interacting channels
    (2, 9, 5, 4.0, True, True),
])
def test_lanes_per_pair_match_one_thread(gpu_ctx, C, T, maxc, cut, block, inter):
    sm = _model(C, block, inter, True)
    ds = random_dye_seqs(120, C, 8, 30, max_per_channel=maxc, seed=C * 7 + T)
    rads, _ = simulate_radiometries(sm, ds, T, 37, seed=C + T)
    gpu_ctx.upload_model(sm, T)
    gpu_ctx.upload_peptides(ds)
    try:
        gpu_ctx.set_engine_config((64, 1, 64, 1))  # one pass, one thread per pair
        one = gpu_ctx.loglik_all(rads, cut)
        # default shapes, and a first slab so small that most pairs pass on
        for cfg in (None, (256, 4, 256, 4)):
            gpu_ctx.set_engine_config(cfg)
            got = gpu_ctx.loglik_all(rads, cut)
            assert np.array_equal(got, one), (cfg, np.sum(got != one), got.size)
    finally:
        gpu_ctx.set_engine_config(None)


@pytest.mark.parametrize("block", [False, True])
def test_dense_slab_classes_vs_oracle(gpu_ctx, oracle, block):
    """Pairs past every pass's slab, of both slab classes of the dense kernel
    (36 to 216 states per Edman slice; the small class ends below 100), in
    one batch."""
    sm = _model(3, block)
    seqs = ["0" * a + "1" * b + "." * 3 + "2" * c for a, b, c in
            [(3, 2, 2), (3, 3, 2), (3, 3, 3), (4, 3, 3), (5, 3, 3), (5, 4, 3), (5, 5, 5), (2, 5, 5), (1, 1, 0)]]
    ds = DyeSeqSet(3, [parse_dye_seq(x) for x in seqs], np.arange(len(seqs), dtype=np.int32),
                   np.ones(len(seqs), np.int32))
    rads, _ = simulate_radiometries(sm, ds, 16, 6, seed=5)
    gpu_ctx.upload_model(sm, 16)
    gpu_ctx.upload_peptides(ds)
    g = gpu_ctx.loglik_all(rads, DBL_MAX)
    assert gpu_ctx.last_batch_stats()["dense"] > 0
    o = oracle.loglik_all(sm, 16, ds, rads, DBL_MAX, threads=8)
    assert_logp_close(g, o, "dense classes")


@pytest.mark.parametrize("block,cut", [(False, DBL_MAX), (True, 4.0)])
def test_passes_side_by_side(gpu_ctx, block, cut):
    """A batch large enough for its passes to run side by side (65,536 pairs):
    read by read the numbers of smaller batches, run directly and as a replayed
    graph."""
    import torch
    sm = _model(3, block)
    ds = random_dye_seqs(110, 3, 8, 26, max_per_channel=4, min_total=1, seed=11)
    rads, _ = simulate_radiometries(sm, ds, 12, 700, seed=12)
    R = len(rads)  # some reads are not detectable
    assert R * 110 >= 65536
    gpu_ctx.upload_model(sm, 12)
    gpu_ctx.upload_peptides(ds)
    whole = gpu_ctx.classify(rads, cut)
    for lo in (0, 350):
        for a, b in zip(gpu_ctx.classify(rads[lo:lo + 350], cut), whole):
            assert np.array_equal(a, b[lo:lo + 350])
    d = torch.from_numpy(rads).cuda()
    oid = torch.zeros(R, dtype=torch.int32, device="cuda")
    osc, otot = (torch.zeros(R, dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    for _ in range(4):
        oid.zero_()
        osc.zero_()
        torch.cuda.synchronize()
        gpu_ctx.classify_device(d.data_ptr(), R, cut, oid.data_ptr(), osc.data_ptr(), otot.data_ptr(), async_=False)
        assert np.array_equal(oid.cpu().numpy(), whole[0]) and np.array_equal(osc.cpu().numpy(), whole[1])
