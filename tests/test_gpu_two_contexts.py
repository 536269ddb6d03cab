"""Two contexts on one device, each in its own thread, with calls whose kernels take
different amounts of shared memory: a launch's shared memory is allowed by an
attribute of the kernel that both contexts share, so it must not shrink under a
launch.  Every call has to succeed with the results it has alone, bit for bit."""
import ctypes
import threading

import numpy as np
import pytest

from whatprot_gb300 import capi
from whatprot_gb300.io import DyeTrackSet
from whatprot_gb300.model import DyeSeqSet, parse_dye_seq
from whatprot_gb300.simulate import paper_model, simulate_radiometries

pytestmark = pytest.mark.gpu


def _together(calls, times):
    """Each call `times` times in a thread of its own, against its result alone."""
    want = [call() for call in calls]
    errors = []
    start = threading.Barrier(len(calls))

    def work(call, first):
        start.wait()
        try:
            for _ in range(times):
                for x, y in zip(call(), first):
                    assert np.array_equal(x, y)
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c, w)) for c, w in zip(calls, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.fixture
def two():
    ctxs = [capi.Context(0), capi.Context(0)]
    yield ctxs
    for c in ctxs:
        c.close()


def test_fits(two):
    def call(ctx, T, s):
        C = 3
        sm, seq = paper_model(C), parse_dye_seq(s)
        ds = DyeSeqSet(C, [seq], np.array([0], np.int32), np.array([1], np.int32))
        rads, _ = simulate_radiometries(sm, ds, T, 60, seed=T)
        ctx.upload_model(sm, T)
        ctx.fit_begin(seq, rads)
        sums, lp, nz = capi.WpFitSums(), ctypes.c_double(0), ctypes.c_int(0)
        f, args = ctx.lib.wp_fit_estep, (ctx.h, ctypes.byref(sums), ctypes.byref(lp), ctypes.byref(nz))

        def go():  # E-steps in quick succession (they take turns otherwise)
            for _ in range(200):
                assert f(*args) == 0, ctx.lib.wp_last_error(ctx.h)
            d = sums.as_dict(T, C)
            return [np.asarray(d[k]) for k in sorted(d)] + [np.float64(lp.value), np.int64(nz.value)]
        return go

    _together([call(two[0], 16, "..0.1.2.0.0.1.2.1.02"), call(two[1], 6, "0.1")], 30)


def test_knn(two):
    T, C = 6, 2

    def call(ctx, ids):
        rng = np.random.default_rng(ids)
        t = np.maximum(rng.integers(0, 6, (600, 1, C)) - np.cumsum(rng.random((600, T, C)) < 0.3, axis=1), 0)
        t = np.unique(t.reshape(600, -1), axis=0).astype(np.int16).reshape(-1, T, C)
        S = max(len(t), ids)
        off = np.minimum(np.arange(len(t) + 1), S).astype(np.int32)
        off[-1] = S
        dts = DyeTrackSet(t, off, (np.arange(S) % ids).astype(np.int32), np.ones(S, np.int32), np.ones(S, np.int32))
        reads = t[rng.integers(0, len(t), 20)] + rng.normal(0, 0.2, (20, T, C))
        ctx.upload_model(paper_model(C), T)
        ctx.upload_tracks(dts)
        return lambda: [x[:, :1] if x.ndim == 2 else x for x in ctx.nn_classify(reads, 50, 0.5, 8)]

    _together([call(two[0], 12000), call(two[1], 10)], 1000)


def test_training(two):
    import torch
    T, C, B = 6, 2, 64

    def call(ctx, P):
        seqs = [np.array([i % 2, -1, (i // 2) % 2], np.int16) for i in range(P)]
        ctx.upload_model(paper_model(C), T)
        ctx.upload_peptides(DyeSeqSet(C, seqs, np.arange(P, dtype=np.int32), np.ones(P, np.int32)))
        net = capi.ProposalNet(ctx, hidden=64, seed=5)
        x = torch.linspace(0, 3, B * T * C, device="cuda").reshape(B, T * C).contiguous()
        y = (torch.arange(B, device="cuda") % P).to(torch.int32)
        torch.cuda.synchronize()

        def go():
            loss = net.train_step(x.data_ptr(), y.data_ptr(), B, 0.0)
            return [np.float64(loss), net.get(5, grad=True)]
        return go

    _together([call(two[0], 30000), call(two[1], 100)], 1500)
