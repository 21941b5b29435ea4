"""GPU tests of the FP32 CUDA-core GEMM's last partial wave (csrc/sgemm.cu): the
tiles beyond whole waves of two CTAs per SM run as K slices and a reduction of
their own.  Ragged tile edges, K not a multiple of the block, every transpose
pair, aligned and unaligned operands; C padding untouched."""
import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("m,n,k,pad", [
    (128 * 25 - 3, 128 * 12 + 5, 700, 0),    # 325 tiles: 29 beyond one wave of 296, 2 slices
    (128 * 30, 128 * 10, 4096, 4),           # 300: 4 tiles in 8 slices
    (128 * 20 + 1, 128 * 21 - 127, 515, 1),  # 441: 145 tiles in 2 slices, odd strides
    (128 * 25, 128 * 24, 255, 0),            # 600: 8 tiles, K too short to slice
])
def test_last_wave_in_slices(cuda, ta, tb, m, n, k, pad):
    import torch

    g = torch.Generator(device=cuda).manual_seed(m + n + k)
    ar, ac = (m, k) if ta == "N" else (k, m)
    br, bc = (k, n) if tb == "N" else (n, k)
    mk = lambda r, c: torch.rand(c, r + pad, device=cuda, generator=g) * 2 - 1  # noqa: E731
    A, B, C0 = mk(ar, ac), mk(br, bc), mk(m, n)
    a, b = A[:, :ar].t().double(), B[:, :br].t().double()
    a, b = (a if ta == "N" else a.t()), (b if tb == "N" else b.t())
    for beta in (0.0, 0.5):
        C = C0.clone()
        torch.cuda.synchronize()
        blas.sgemm_device(ta, tb, m, n, k, 1.5, A, ar + pad, B, br + pad, beta, C, m + pad)
        torch.cuda.synchronize()
        ref = 1.5 * (a @ b) + beta * C0[:, :m].t().double()
        bar = 8 * k * 2.0 ** -24 * 1.5 * float(a.norm()) * float(b.norm())
        assert float((C[:, :m].t().double() - ref).norm()) <= bar
        assert torch.equal(C[:, m:], C0[:, m:]), "padding rows of C were written"
