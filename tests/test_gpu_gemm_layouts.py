"""Products whose operands are stored with the reduction dimension as rows, as
the proposal network's backward pass takes them, at the sizes where a tile
ends: one training step's gradients for hidden widths and batches at and
beside the tile sizes (narrow tiles where a gradient has few), against the
FP64 oracle with the GPU's BF16 roundings.  Tolerance as test_gpu_mlp.py (1e-3
relative Frobenius error)."""
import os
import sys

import numpy as np
import pytest

from whatprot_gb300 import capi
from whatprot_gb300.model import DyeSeqSet
from whatprot_gb300.simulate import paper_model

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))


@pytest.mark.parametrize("B,P,hidden", [(64, 200, 192), (320, 700, 256), (128, 20000, 320), (64, 129, 1088)])
def test_gradients_by_layout(gpu_ctx, B, P, hidden):
    import torch
    import mlp_oracle
    T, C = 8, 2
    seqs = [np.array([i % 2, -1, (i // 2) % 2], np.int16) for i in range(P)]
    gpu_ctx.upload_model(paper_model(C), T)
    gpu_ctx.upload_peptides(DyeSeqSet(C, seqs, np.arange(P, dtype=np.int32), np.ones(P, np.int32)))
    net = capi.ProposalNet(gpu_ctx, hidden=hidden, seed=9)
    g = torch.Generator(device="cuda")
    g.manual_seed(B + P + hidden)
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
