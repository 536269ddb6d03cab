"""One training step at the sizes where its memory passes (logit-gradient
softmax, transposes, column sums) change shape: the smallest batch and class
count, a row that no longer fits shared memory, class counts at and beside a
multiple of 64.  Loss and gradients against the FP64 oracle with the GPU's
BF16 roundings, at the tolerances of test_gpu_mlp.py (1e-3 relative Frobenius
error: the gradients are sums of BF16-rounded terms; bias gradients are FP32
sums of at most 256 such terms, whose rounding is far below that)."""
import os
import sys

import numpy as np
import pytest

from whatprot_gb300 import capi
from whatprot_gb300.model import DyeSeqSet
from whatprot_gb300.simulate import paper_model

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))


@pytest.mark.parametrize("B,P,hidden", [(64, 1, 64), (64, 63, 64), (192, 65, 128), (256, 1000, 64), (64, 57000, 64)])
def test_step_gradients(gpu_ctx, B, P, hidden):
    import torch
    import mlp_oracle
    T, C = 8, 2
    seqs = [np.array([i % 2, -1, (i // 2) % 2], np.int16) for i in range(P)]
    gpu_ctx.upload_model(paper_model(C), T)
    gpu_ctx.upload_peptides(DyeSeqSet(C, seqs, np.arange(P, dtype=np.int32), np.ones(P, np.int32)))
    net = capi.ProposalNet(gpu_ctx, hidden=hidden, seed=5)
    g = torch.Generator(device="cuda")
    g.manual_seed(B + P)
    x = torch.rand(B, T * C, generator=g, device="cuda") * 3
    y = torch.randint(-1, P, (B,), generator=g, device="cuda", dtype=torch.int32)
    loss = net.train_step(x.data_ptr(), y.data_ptr(), B, 0.0)
    w = {n: net.get(i).astype(np.float64) for i, n in enumerate(net.PARAMS)}
    o_loss, o_grad, _ = mlp_oracle.gradients(w, x.cpu().numpy().astype(np.float64), y.cpu().numpy(), P)
    assert abs(loss - o_loss) <= 3e-4 * abs(o_loss) + 1e-6
    for i, n in enumerate(net.PARAMS):
        got, want = net.get(i, grad=True).astype(np.float64).reshape(o_grad[n].shape), o_grad[n]
        err = np.linalg.norm(got - want)
        assert err <= 1e-3 * np.linalg.norm(want) + 1e-7, (n, err, np.linalg.norm(want))
    net.close()
