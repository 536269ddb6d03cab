"""E-steps with a read whose dyes of one channel go dark for some cycles and come
back: an ordinary fault of a real run (a missed registration, a blinking dye)
that the model gives a small, positive probability.  The forward vector then
holds the read's only path at 2^-33 or so per dark dye and cycle, and the frame
factor of its counts is the inverse.

Every sum has to be finite, alone and among clean reads, and with the warp
kernel no further from the oracle than with the thread-per-read kernel, up to
the 1e-5 of the parameter's denominator that test_gpu_fit.py allows any E-step
(both hold the vectors in FP32: a path far enough below the largest entry is lost
to both, below 2^-149 to the thread kernel).  While dark dyes times cycles are at
most two (2^-66), nothing is lost: 1e-5."""
import numpy as np
import pytest

from oracle_lib import WpoFitSums
from whatprot_gb300.model import DyeSeqSet, parse_dye_seq
from whatprot_gb300.simulate import paper_model, simulate_radiometries

pytestmark = pytest.mark.gpu

CONTROL = "..0.1.2.0.0.1.2.1.02"  # 4 / 3 / 3 dyes
CASES = [
    # C, T, dye-seq, dark channel, dark cycles, blocking, emission
    (3, 16, CONTROL, 0, 1, False, True),
    (3, 16, CONTROL, 0, 2, False, True),
    (3, 16, CONTROL, 1, 2, False, False),
    (3, 16, CONTROL, 2, 2, True, False),
    (3, 16, CONTROL, 1, 3, True, True),
    (3, 16, CONTROL, 2, 5, False, False),
    (1, 9, ".......0", 0, 1, False, True),
    (1, 9, ".......0", 0, 3, False, True),
    (1, 9, ".......0", 0, 4, False, True),   # the largest entry is subnormal afterwards
    (1, 9, ".......0", 0, 4, True, False),
    (1, 12, "........0", 0, 5, False, True),
    (2, 10, "......0.0.1", 0, 2, False, True),
    (2, 10, "......0.0.01", 0, 2, True, True),
    (2, 10, "......0.0.0.01", 0, 1, False, False),
    (2, 10, "......0.0.0.0.01", 0, 1, True, False),
]


def _blinking(sm, C, T, seq, channel, dark):
    """A read without losses but the cut's, channel `channel` dark from cycle 1."""
    x = np.zeros((1, T, C))
    for t in range(T):
        for c in range(C):
            n = int((seq[t:] == c).sum())
            x[0, t, c] = n + 0.02 * n * (-1) ** (t + c) + 0.002
    x[0, 1:1 + dark, channel] = 0.003
    return x


@pytest.mark.parametrize("clean", [0, 200])
@pytest.mark.parametrize("case", CASES, ids=[f"C{c[0]}T{c[1]}n{len(c[2])}c{c[3]}x{c[4]}{'B' if c[5] else ''}{'E' if c[6] else ''}" for c in CASES])
def test_blinking_read(gpu_ctx, oracle, case, clean):
    C, T, s, channel, dark, block, emission = case
    sm = paper_model(C)
    if block:
        sm.p_initial_block, sm.p_cyclic_block = 0.04, 0.03
    seq = parse_dye_seq(s)
    bad = _blinking(sm, C, T, np.asarray(seq), channel, dark)
    ds = DyeSeqSet(C, [seq], np.array([0], np.int32), np.array([1], np.int32))
    good, _ = simulate_radiometries(sm, ds, T, 2 * clean + 20, seed=T + dark)
    rads = np.concatenate([good[:clean // 2], bad, good[clean // 2:clean]])
    gpu_ctx.upload_model(sm, T)
    gpu_ctx.fit_begin(seq, rads)
    gpu_ctx.fit_set_emission(emission)
    got = []
    try:
        for kind in (0, 1):
            gpu_ctx.fit_set_kernel(kind)
            sums, lp, nz = gpu_ctx.fit_estep()
            d = sums.as_dict(T, C)
            if emission:
                d.update(zip(("emis_w", "emis_x", "emis_xx"), gpu_ctx.fit_emission_sums().arrays(C)))
            assert np.isfinite(lp) or nz == len(rads)
            for k, v in d.items():
                assert np.all(np.isfinite(v)), (kind, k, v)
            got.append((d, nz))
    finally:
        gpu_ctx.fit_set_kernel(0)
        gpu_ctx.fit_set_emission(False)
    (a, nza), (b, nzb) = got
    assert nza <= nzb
    o = WpoFitSums()
    for r in rads:
        oracle.improve_fit(sm, T, seq, r, max(int((seq == c).sum()) for c in range(C)), sums=o)
    e = o.as_dict(T, C)
    lost = int((np.asarray(seq)[1:] == channel).sum()) * dark > 2

    def near(key, want, den):
        x, y, w = (np.asarray(v, np.float64) for v in (a[key], b[key], want))
        tol = 1e-5 * np.maximum(np.asarray(den, np.float64), 1e-3)
        assert np.all(np.abs(x - w) <= (np.abs(y - w) if lost else 0.0) + tol), (key, x, y, w)

    for k in ("edman", "bleach", "dud", "init_block", "cyc_block"):
        near(k + "_num", e[k][0], e[k][1])
        near(k + "_den", e[k][1], e[k][1])
    near("detach_n", e["detach_n"], e["detach_n"])
    near("detach_x", e["detach_x"], e["detach_n"])
    if emission:
        for k in ("emis_w", "emis_x", "emis_xx"):
            near(k, e[k], np.full_like(e[k], e["emis_w"].sum() / C))


FAR = [
    # C, T, dye-seq, dark channel, from cycle, dark cycles.  Kernel 0 is the warp kernel, and
    # for the second shape (110 states, 44 timesteps) the CTA kernel.
    (1, 60, "." * 56 + "0", 0, 1, 40),
    (2, 44, "0" * 8 + "1" * 10 + "." * 30 + "0", 0, 8, 35),
]


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("case", FAR, ids=["C1T60", "C2T44"])
def test_frame_beyond_fp64(gpu_ctx, case, kind):
    """Forward and backward vectors whose overlap is below 2^-1023, the end of an
    FP64 factor: finite sums (the read's own counts have underflowed)."""
    C, T, s, channel, start, dark = case
    sm = paper_model(C)
    seq = np.asarray(parse_dye_seq(s))
    x = _blinking(sm, C, T, seq, channel, 0)
    x[0, start:start + dark, channel] = 0.003
    gpu_ctx.upload_model(sm, T)
    gpu_ctx.fit_begin(seq, x)
    gpu_ctx.fit_set_emission(True)
    gpu_ctx.fit_set_kernel(kind)
    try:
        sums, lp, nz = gpu_ctx.fit_estep()
        em = gpu_ctx.fit_emission_sums().arrays(C)
    finally:
        gpu_ctx.fit_set_kernel(0)
        gpu_ctx.fit_set_emission(False)
    assert nz == 0 and np.isfinite(lp)
    for k, v in sums.as_dict(T, C).items():
        assert np.all(np.isfinite(v)), (k, v)
    for v in em:
        assert np.all(np.isfinite(v))


@pytest.mark.parametrize("kind", [0, 1])
def test_subnormal_largest_entry(gpu_ctx, oracle, kind):
    """One dye dark for four cycles and nearly so for a fifth: the vector left has its
    largest entry near 2^-138, beyond 2^-127 which one FP32 factor undoes, and with 11
    bits there (the warp kernel holds it higher).  Some ten roundings of 2^-12 in a row:
    2.5e-3 of a count; 1e-2 allowed."""
    C, T = 1, 10
    sm = paper_model(C)
    seq = np.asarray(parse_dye_seq("........0"))
    x = _blinking(sm, C, T, seq, 0, 4)
    x[0, 5, 0] = 0.038
    gpu_ctx.upload_model(sm, T)
    gpu_ctx.fit_begin(seq, x)
    gpu_ctx.fit_set_kernel(kind)
    try:
        sums, _, _ = gpu_ctx.fit_estep()
    finally:
        gpu_ctx.fit_set_kernel(0)
    a = sums.as_dict(T, C)
    _, _, o = oracle.improve_fit(sm, T, seq, x[0], 1)
    e = o.as_dict(T, C)
    for k in ("edman", "bleach", "dud", "cyc_block"):
        for j, w in enumerate(("_num", "_den")):
            assert np.all(np.abs(a[k + w] - np.asarray(e[k][j])) <= 1e-2 * np.maximum(e[k][1], 1e-3)), (k + w, a[k + w], e[k][j])
    assert np.all(np.abs(a["detach_n"] - e["detach_n"]) <= 1e-2), (a["detach_n"], e["detach_n"])
