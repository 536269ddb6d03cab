"""Kept launch shapes (wp_shape.cu) against what they depend on: a device reset takes
the functions' attributes with it, and a context made after it must ask again.  In a
child process, whose own CUDA context alone the reset ends."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes, sys
sys.path[:0] = [%(repo)r, %(repo)r + "/tests"]
import numpy as np
from whatprot_gb300 import capi
from whatprot_gb300.simulate import paper_model, random_dye_seqs, simulate_radiometries
from test_zz_no_alloc import _bind, _model_struct

sm, T = paper_model(3), 12
ds = random_dye_seqs(70, 3, 8, 24, max_per_channel=5, min_total=1, seed=3)
rads, _ = simulate_radiometries(sm, ds, T, 60, seed=4)
lib = capi.load_library()
cudart = ctypes.CDLL(%(cudart)r)


def kept():
    ctx = capi.Context(0)
    ctx.upload_model(sm, T)
    ctx.upload_peptides(ds)
    out = ctx.classify(rads, 5.0)
    ctx.close()
    return out


def noalloc():
    m, keep = _model_struct(sm)
    flat, off = ds.ragged()
    R = len(rads)
    out = [np.zeros(R, np.int32), np.zeros(R), np.zeros(R)]
    assert _bind(lib)(0, ctypes.byref(m), T, flat.ctypes.data, off.ctypes.data, ds.ids.ctypes.data,
                      ds.counts.ctypes.data, len(ds), rads.ctypes.data, R, 5.0, *[o.ctypes.data for o in out]) == 0
    return out


a = kept()
b = noalloc() if %(alone)d else None
for again in range(2):
    assert cudart.cudaDeviceReset() == 0
    for x, y in zip(a, kept()):
        assert np.array_equal(x, y)
print("same")
"""


def _cudart():
    for line in subprocess.run(["ldd", os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "whatprot_gb300",
                                                    "_lib", "libwhatprot_gb300.so")], capture_output=True,
                               text=True).stdout.splitlines():
        if "libcudart" in line:
            return line.split("=>")[1].split()[0]
    pytest.skip("the library carries its own CUDA runtime")


@pytest.mark.parametrize("alone", [0, 1])
def test_device_reset(alone):
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = CHILD % {"repo": repo, "cudart": _cudart(), "alone": alone}
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
