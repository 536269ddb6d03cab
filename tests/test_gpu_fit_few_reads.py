"""Which E-step kernel takes few reads and which many (a channel of many dyes, long
blocked chains), and that both give the same sums: one E-step over all reads against
the E-steps over a dozen parts of them.  Each kernel is within 1e-5 of the oracle by
test_gpu_fit.py's rule, so the two are within 2e-5 of each other."""
import numpy as np
import pytest

from whatprot_gb300.model import DyeSeqSet
from whatprot_gb300.simulate import paper_model, simulate_radiometries

pytestmark = pytest.mark.gpu

CASES = [
    # T, dyes per channel, blocking, kernel for 100 and for 1,200 reads
    (12, (5,), False, "warp", "warp"),
    (12, (6,), False, "warp", "warp"),
    (12, (6,), True, "cta", "warp"),
    (33, (6,), False, "cta", "warp"),
    (8, (6, 6), False, "cta", "warp"),
    (9, (7, 7), True, "cta", "warp"),
    (10, (2, 6, 1), True, "cta", "warp"),
    (40, (2,), True, "warp", "warp"),
    (41, (2,), True, "cta", "warp"),
    (41, (2,), False, "warp", "warp"),
    (20, (13,), True, "cta", "warp"),
    (41, (13,), True, "cta", "cta"),
    (41, (13,), False, "cta", "warp"),
]


@pytest.mark.parametrize("T,dyes,block,few,many", CASES,
                         ids=[f"T{c[0]}n{'.'.join(map(str, c[1]))}{'B' if c[2] else ''}" for c in CASES])
def test_parts_and_whole(gpu_ctx, T, dyes, block, few, many):
    C, R, part = len(dyes), 1200, 100
    sm = paper_model(C)
    if block:
        sm.p_initial_block, sm.p_cyclic_block = 0.03, 0.03
    seq = np.random.default_rng(T).permutation(np.repeat(np.arange(C), dyes)).astype(np.int16)
    ds = DyeSeqSet(C, [seq], np.zeros(1, np.int32), np.ones(1, np.int32))
    rads = simulate_radiometries(sm, ds, T, 2 * R, seed=T)[0][:R]
    assert len(rads) == R
    gpu_ctx.upload_model(sm, T)

    def estep(x):
        gpu_ctx.fit_begin(seq, x)
        s, lp, nz = gpu_ctx.fit_estep()
        return {k: np.asarray(v, np.float64) for k, v in s.as_dict(T, C).items()}, lp, nz

    whole, lp, nz = estep(rads)
    assert gpu_ctx.last_routes()["estep"] == many
    parts = []
    for r0 in range(0, R, part):
        parts.append(estep(rads[r0:r0 + part]))
        assert gpu_ctx.last_routes()["estep"] == few
    assert nz == sum(p[2] for p in parts)
    assert np.isclose(lp, sum(p[1] for p in parts), rtol=2e-5)
    total = {k: sum(p[0][k] for p in parts) for k in whole}
    den = {"detach_x": "detach_n"}
    for k in whole:
        d = total[den.get(k, k.replace("_num", "_den"))]
        assert np.all(np.abs(whole[k] - total[k]) <= 2e-5 * np.maximum(d, 1e-3)), k


def test_batch(gpu_ctx):
    """Lists of reads share the resident CTAs: five lists of 100 are more than a turn."""
    sm = paper_model(1)
    sm.p_cyclic_block = 0.03
    seq = np.zeros(7, np.int16)
    ds = DyeSeqSet(1, [seq], np.zeros(1, np.int32), np.ones(1, np.int32))
    rads = simulate_radiometries(sm, ds, 10, 300, seed=1)[0][:100]
    gpu_ctx.upload_model(sm, 10)
    gpu_ctx.fit_begin(seq, rads)
    idx = np.arange(100)
    for B, want in ((1, "cta"), (50, "warp")):
        s, lp, nz = gpu_ctx.fit_estep_batch([sm] * B, np.tile(idx, (B, 1)))
        assert gpu_ctx.last_routes()["estep"] == want
        one = gpu_ctx.fit_estep()
        a, b = s[-1].as_dict(10, 1), one[0].as_dict(10, 1)
        assert np.allclose(a["bleach_den"], b["bleach_den"], rtol=2e-5)
        assert np.allclose(a["edman_num"], b["edman_num"], rtol=2e-5)
