"""The batch's preparation (emission ranges and factors, the reads' boxes, the
window factors) where whole reads fill a CTA differently: one timestep, numbers
of timesteps that do not divide the CTA, the longest; read counts beside a full
CTA.  Log-likelihoods against the oracle at the tolerance of
test_gpu_forward.py."""
import numpy as np
import pytest

from oracle_lib import DBL_MAX
from test_gpu_forward import _model, assert_logp_close
from whatprot_gb300.simulate import random_dye_seqs, simulate_radiometries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,C", [(1, 2), (5, 3), (17, 1), (33, 2), (50, 1), (64, 2)])
@pytest.mark.parametrize("cut", [5.0, DBL_MAX])
def test_preparation_by_timesteps(gpu_ctx, oracle, T, C, cut):
    sm = _model(C)
    ds = random_dye_seqs(6, C, max(3, T // 2), T + 5, max_per_channel=2, min_total=1, seed=T)
    per_cta = 128 // T
    rads, _ = simulate_radiometries(sm, ds, T, 4 * per_cta + 40, seed=T + C)
    gpu_ctx.upload_model(sm, T)
    gpu_ctx.upload_peptides(ds)
    for R in sorted({1, per_cta, per_cta + 1, min(len(rads), 2 * per_cta + 3)}):
        if R > min(len(rads), 300):
            continue
        g = gpu_ctx.loglik_all(rads[:R], cut)
        o = oracle.loglik_all(sm, T, ds, rads[:R], cut, threads=8)
        assert_logp_close(g, o, (T, C, cut, R))
