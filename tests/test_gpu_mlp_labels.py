"""A label that is no class of the network (a stale one from a larger peptide set):
an error, with nothing written outside the example's own place.  The example
counts as one to skip, so the gradients are those with -1 in its place, bit for
bit, and the weights stay as they are.  With the row of logits in shared memory
and, beyond 56,000 classes, read again for each pass."""
import numpy as np
import pytest

from whatprot_gb300 import capi
from whatprot_gb300.model import DyeSeqSet
from whatprot_gb300.simulate import paper_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,label", [(65, 65), (65, 127), (65, 128), (65, 2 ** 31 - 1), (64, 64), (57000, 57000)])
def test_label_without_class(gpu_ctx, P, label):
    import torch
    T, C, B = 8, 2, 64
    seqs = [np.array([i % 2, -1, (i // 2) % 2], np.int16) for i in range(P)]
    gpu_ctx.upload_model(paper_model(C), T)
    gpu_ctx.upload_peptides(DyeSeqSet(C, seqs, np.arange(P, dtype=np.int32), np.ones(P, np.int32)))
    net = capi.ProposalNet(gpu_ctx, hidden=64, seed=5)
    g = torch.Generator(device="cuda")
    g.manual_seed(P)
    x = torch.rand(B, T * C, generator=g, device="cuda") * 3
    y = torch.randint(0, P, (B,), generator=g, device="cuda", dtype=torch.int32)
    y[B - 1] = -1
    net.train_step(x.data_ptr(), y.data_ptr(), B, 0.0)
    want = [net.get(i, grad=True) for i in range(6)]
    weights = [net.get(i) for i in range(6)]
    y[B - 1] = label
    for lr in (0.0, 1e-3):
        with pytest.raises(capi.WpError) as e:
            net.train_step(x.data_ptr(), y.data_ptr(), B, lr)
        assert e.value.status == 1  # WP_ERR_INVALID
        for i in range(6):
            assert np.array_equal(net.get(i, grad=True), want[i]), i
            assert np.array_equal(net.get(i), weights[i]), i
    y[B - 1] = P - 1
    assert np.isfinite(net.train_step(x.data_ptr(), y.data_ptr(), B, 1e-3))  # and the network goes on
    assert not np.array_equal(net.get(4), weights[4])
    net.close()
