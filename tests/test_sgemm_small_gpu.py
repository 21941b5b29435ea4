"""GPU tests of the FP32 kernel's 64x64 form (csrc/sgemm.cu): tile and K-panel
edges, one and several K slices, every transpose pair, leading dimensions that
take 16-byte and 4-byte copies, element by element against FP64 products of the
same inputs; surroundings of the operands hold NaN, C's padding stays."""
import numpy as np
import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu
SHAPES = [(1, 1, 1), (63, 65, 15), (64, 64, 16), (65, 63, 17), (100, 200, 70), (129, 60, 513),
          (40, 33, 4099), (320, 130, 1030)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("off,pad", [(0, 0), (1, 3), (4, 4)])
def test_small_products(cuda, m, n, k, off, pad):
    import torch

    rng = np.random.default_rng(m + 10 * n + 100 * k)
    st = torch.cuda.Stream()

    def operand(rows, cols, ld):
        buf = np.full(off + ld * cols + 8, np.nan, np.float32)
        view = buf[off:off + ld * cols].reshape(cols, ld)
        view[:, :rows] = rng.uniform(-1, 1, (cols, rows)).astype(np.float32)
        return torch.from_numpy(buf).to(cuda), view[:, :rows].astype(np.float64).T

    up = (lambda x: (x + 3) // 4 * 4) if off % 4 == 0 and pad == 4 else (lambda x: x)
    for ta in "NT":
        for tb in "NT":
            ar, ac = (m, k) if ta == "N" else (k, m)
            br, bc = (k, n) if tb == "N" else (n, k)
            lda, ldb, ldc = up(ar) + pad, up(br) + pad, m + pad
            (da, a), (db, b), (dc, c) = operand(ar, ac, lda), operand(br, bc, ldb), operand(m, n, ldc)
            torch.cuda.synchronize()
            blas.sgemm_device(ta, tb, m, n, k, 1.25, da[off:], lda, db[off:], ldb, -0.5, dc[off:],
                              ldc, method="fp32", stream=st)
            torch.cuda.synchronize()
            oa, ob = (a if ta == "N" else a.T), (b if tb == "N" else b.T)
            after = dc.cpu().numpy()
            got = after[off:off + ldc * n].reshape(n, ldc)
            assert np.isnan(got[:, m:]).all() and np.isnan(after[:off]).all()
            assert np.isnan(after[off + ldc * n:]).all()
            # k products and sums in FP32, the scaling and the final add
            bound = (k + 4) * 2.0 ** -24 * (1.25 * (np.abs(oa) @ np.abs(ob)) + np.abs(c))
            err = np.abs(got[:, :m].T.astype(np.float64) - (1.25 * (oa @ ob) - 0.5 * c))
            assert (err <= bound).all(), (ta, tb)


@pytest.mark.parametrize("m,n,k", [(384, 240, 848), (3072, 3072, 512)])
def test_captured_calls_hold_no_scratch(cuda, m, n, k):
    """A captured call allocates nothing, and its graph stays right after a
    larger call has replaced the scratch that running calls slice K with."""
    import torch

    def product(rows, cols, inner, st):
        a, b = (torch.rand(x, device=cuda) for x in (rows * inner, inner * cols))
        c = torch.zeros(rows * cols, device=cuda)
        call = lambda: blas.sgemm_device("N", "N", rows, cols, inner, 1.0, a, rows, b, inner, 0.0, c,  # noqa: E731
                                         rows, method="fp32", stream=st)
        return a, b, c, call

    st = torch.cuda.Stream()
    a, b, c, call = product(m, n, k, st)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(st):
        with torch.cuda.graph(graph, stream=st):
            call()
    big = product(4096, 4096, 1024, st)
    torch.cuda.synchronize()
    big[3]()
    graph.replay()
    torch.cuda.synchronize()
    ref = a.view(k, m).double().T @ b.view(n, k).double().T
    err = (c.view(n, m).T.double() - ref).abs().max()
    assert err <= (k + 4) * 2.0 ** -24 * ref.max()  # all operands are positive
