"""The warp-per-read E-step (wp_fitw.cu) against the thread-per-read kernel and
the oracle, at the shapes where it changes route: one to four channels, a
channel without dyes, fibres longer than its registers hold, S of 1 and around
a multiple of 32, one timestep, blocking, emission statistics, more reads than
resident warps.

Both sides form FP32 terms of positive sums and add them over reads in FP64.
A term carries the rounding of its two vectors, at most about 6 T roundings of
2^-24 in a chain of T timesteps (detachment, bleach steps, cut, emission and
the scale): 6 x 16 x 6e-8 = 6e-6 for a read, less for their sum.  Tolerance
1e-5 of each parameter's denominator, as the package's other E-step tests."""
import numpy as np
import pytest

from oracle_lib import WpoFitSums
from whatprot_gb300.model import DyeSeqSet, parse_dye_seq
from whatprot_gb300.simulate import paper_model, simulate_radiometries

pytestmark = pytest.mark.gpu

CASES = [
    # C, T, dye-seq, reads, blocking, emission
    (1, 8, "0..0.", 40, False, True),
    (2, 1, "01.0", 40, False, True),          # one timestep
    (2, 9, ".0..0", 40, False, False),        # channel 1 without dyes
    (2, 12, "0101010..01", 60, True, True),   # S = 30, blocking
    (3, 16, "..0.1.2.0.0.1.2.1.02", 60, False, True),
    (3, 16, "..0.1.2.0.0.1.2.1.02", 40, True, False),
    (4, 10, "0123.0.3", 40, False, False),    # four channels
    (1, 14, "0000000.0000", 40, False, True), # eleven dyes on a channel: a fibre of twelve
    (2, 6, "", 10, False, False),             # no dyes: S = 1
    (2, 7, "0.1", 9000, False, False),        # several reads per warp
]


@pytest.mark.parametrize("case", CASES, ids=[f"C{c[0]}T{c[1]}{c[2] or 'none'}r{c[3]}{'B' if c[4] else ''}{'E' if c[5] else ''}" for c in CASES])
def test_warp_estep(gpu_ctx, oracle, case):
    C, T, s, reads, block, emission = case
    sm = paper_model(C)
    if block:
        sm.p_initial_block, sm.p_cyclic_block = 0.04, 0.03
    seq = parse_dye_seq(s)
    some = seq if len(seq) else parse_dye_seq("0")
    ds = DyeSeqSet(C, [some], np.array([0], np.int32), np.array([1], np.int32))
    rads, _ = simulate_radiometries(sm, ds, T, int(reads * 1.6) + 20, seed=17 + T)
    rads = rads[:reads]
    if not len(seq):
        rads = np.abs(rads) * 1e-3
    gpu_ctx.upload_model(sm, T)
    gpu_ctx.fit_begin(seq, rads)
    gpu_ctx.fit_set_emission(emission)
    try:
        got = []
        for kind in (0, 1):
            gpu_ctx.fit_set_kernel(kind)
            sums, lp, nz = gpu_ctx.fit_estep()
            got.append((sums.as_dict(T, C), lp, nz, [a.copy() for a in gpu_ctx.fit_emission_sums().arrays(C)]))
    finally:
        gpu_ctx.fit_set_kernel(0)
        gpu_ctx.fit_set_emission(False)
    (a, lpa, nza, ea), (b, lpb, nzb, eb) = got
    assert nza == nzb
    assert abs(lpa - lpb) <= 1e-5 * abs(lpb) + 1e-5

    def close(x, y, den):
        assert np.all(np.abs(np.asarray(x) - np.asarray(y)) <= 1e-5 * np.maximum(np.asarray(den), 1e-3)), (x, y)

    for k in ("edman", "init_block", "cyc_block", "bleach", "dud"):
        close(a[k + "_num"], b[k + "_num"], b[k + "_den"])
        close(a[k + "_den"], b[k + "_den"], b[k + "_den"])
    close(a["detach_x"], b["detach_x"], b["detach_n"])
    close(a["detach_n"], b["detach_n"], b["detach_n"])
    if emission:
        for x, y in zip(ea, eb):
            close(x, y, np.full_like(y, eb[0].sum() / C))
    if reads <= 60:
        o = WpoFitSums()
        most = max([int((seq == c).sum()) for c in range(C)] + [0])
        for r in rads:
            oracle.improve_fit(sm, T, seq, r, most, sums=o)
        d = o.as_dict(T, C)
        for k in ("edman", "bleach", "dud"):
            close(a[k + "_num"], d[k][0], d[k][1])
            close(a[k + "_den"], d[k][1], d[k][1])
        close(a["detach_n"], d["detach_n"], d["detach_n"])
        close(a["detach_x"], d["detach_x"], d["detach_n"])
