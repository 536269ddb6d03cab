"""The GEMM's epilogue stores: 32-byte, 16-byte and element stores by the
alignment of a row, rows and columns past the tiles, and nothing written
outside the product.

Tolerance as in test_gpu_gemm.py: FP32 sums in another order, 1e-4 sqrt(K);
BF16 outputs one rounding (2^-8) besides."""
import ctypes
import math

import pytest

from whatprot_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(1, 1), (33, 31), (128, 256), (130, 288), (97, 513)])
@pytest.mark.parametrize("pad,off", [(0, 0), (4, 0), (8, 4), (16, 8), (3, 1)])
@pytest.mark.parametrize("fp32", [True, False])
def test_gemm_store_alignments(M, N, pad, off, fp32):
    import torch
    K = 64
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + pad)
    A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g)
    ldc = (N + 15) // 16 * 16 + pad
    dt = torch.float32 if fp32 else torch.bfloat16
    buf = torch.full((off + M * ldc + 64,), 7.0, device="cuda", dtype=dt)
    z = torch.full_like(buf, 7.0, dtype=torch.bfloat16)
    lib = capi.load_library()
    P = ctypes.c_void_p
    st = lib.wp_dev_gemm_bf16(P(A.data_ptr()), K, P(B.data_ptr()), K, M, N, K,
                              P(buf.data_ptr() + off * buf.element_size()), ldc, int(fp32), P(bias.data_ptr()), 1,
                              P(z.data_ptr() + off * z.element_size()))
    assert st == 0
    zr = A.float() @ B.float().T + bias
    cr = 0.5 * zr * (1.0 + torch.erf(zr / math.sqrt(2.0)))
    for got, ref, rnd in ((buf, cr, 0.0 if fp32 else 2.0 ** -8), (z, zr, 2.0 ** -8)):
        body = got[off:off + M * ldc].view(M, ldc)
        assert ((body[:, :N].float() - ref).abs() <= 1e-4 * math.sqrt(K) + rnd * ref.abs()).all()
        assert (body[:, N:] == 7.0).all() and (got[:off] == 7.0).all() and (got[off + M * ldc:] == 7.0).all()
