"""GPU tests of the passes that split operands for the tensor cores (csrc/sgemm_tc.cu,
split_kernel and split3m_kernel): bases off a 16-byte (complex: 8-byte) boundary, odd
leading dimensions, edges of the 64 x 64 and 64 x 32 blocks and of the K padding, both
operands in one launch; NaN around the operands, C's padding stays.

Element by element against FP64.  Error of a product relative to |A||B|: the inputs as
they are held (TF32, 11 bits, 2^-11 each; two TF32 2^-22 and the dropped small x small
product as much again; two bfloat16 2^-18 likewise), and one truncation 2^-23 per MMA of
32 bytes of K and term."""
import numpy as np
import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu
INPUT = {"tf32": 2 * 2.0 ** -11, "tf32x3": 3 * 2.0 ** -22, "bf16x3": 3 * 2.0 ** -18}
PER_K = {"tf32": 1 / 8, "tf32x3": 3 / 8, "bf16x3": 3 / 16}


def _operand(cuda, rng, rows, cols, off, ld):
    import torch

    buf = np.full(off + ld * cols + 64, np.nan, np.float32)
    buf[off:off + ld * cols].reshape(cols, ld)[:, :rows] = rng.uniform(-1, 1, (cols, rows))
    view = buf[off:off + ld * cols].reshape(cols, ld)[:, :rows].T.astype(np.float64)
    return torch.from_numpy(buf).to(cuda), view


@pytest.mark.parametrize("method", sorted(INPUT))
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (64, 65, 31), (63, 128, 64), (129, 64, 97),
                                   (200, 333, 129)])
@pytest.mark.parametrize("off,pad", [(0, 0), (1, 0), (4, 1), (2, 4), (0, 3)])
def test_operands_of_any_alignment(cuda, method, ta, tb, m, n, k, off, pad):
    import torch

    rng = np.random.default_rng(m + 10 * n + 100 * k + off)
    ar, ac = (m, k) if ta == "N" else (k, m)
    br, bc = (k, n) if tb == "N" else (n, k)
    da, a = _operand(cuda, rng, ar, ac, off, ar + pad)
    db, b = _operand(cuda, rng, br, bc, (off + 1) % 5, br + pad)
    dc, c = _operand(cuda, rng, m, n, off, m + pad)
    torch.cuda.synchronize()
    blas.sgemm_device(ta, tb, m, n, k, 1.25, da[off:], ar + pad, db[(off + 1) % 5:], br + pad, -0.5,
                      dc[off:], m + pad, method=method)
    torch.cuda.synchronize()
    a, b = (a if ta == "N" else a.T), (b if tb == "N" else b.T)
    after = dc.cpu().numpy()
    got = after[off:off + (m + pad) * n].reshape(n, m + pad)
    assert np.isnan(got[:, m:]).all() and np.isnan(after[:off]).all()
    assert np.isnan(after[off + (m + pad) * n:]).all()
    scale = 1.25 * (np.abs(a) @ np.abs(b))
    bound = (INPUT[method] + (PER_K[method] * k + 2) * 2.0 ** -23) * scale + 2.0 ** -22 * (
        scale + np.abs(c))
    assert (np.abs(got[:, :m].T - (1.25 * (a @ b) - 0.5 * c)) <= bound).all()


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("C", "T"), ("R", "C"), ("T", "R")])
@pytest.mark.parametrize("m,n,k,off", [(257, 260, 255, 1), (300, 190, 330, 2), (64, 4099, 65, 3)])
def test_complex_operands_of_any_alignment(cuda, ta, tb, m, n, k, off):
    """Products of 2^24 multiply-adds and more; bases at any multiple of 4 bytes."""
    import torch

    rng = np.random.default_rng(m + k)

    def operand(rows, cols):
        buf = np.full(off + 2 * rows * cols + 64, np.nan, np.float32)
        x = rng.uniform(-1, 1, 2 * rows * cols).astype(np.float32)
        buf[off:off + x.size] = x
        t = torch.from_numpy(buf).to(cuda)
        return t, t.data_ptr() + 4 * off, x.reshape(cols, rows, 2).astype(np.float64)

    keep = "NR"
    ar, ac = (m, k) if ta in keep else (k, m)
    br, bc = (k, n) if tb in keep else (n, k)
    (ta_, pa, a), (tb_, pb, b), (tc_, pc, c) = operand(ar, ac), operand(br, bc), operand(m, n)
    cx = lambda x: (x[..., 0] + 1j * x[..., 1]).T  # noqa: E731
    op = lambda x, t: {"N": x, "T": x.T, "C": x.conj().T, "R": x.conj()}[t]  # noqa: E731
    a, b, c = op(cx(a), ta), op(cx(b), tb), cx(c)
    torch.cuda.synchronize()
    blas.cgemm3m_device(ta, tb, m, n, k, 0.5 - 0.25j, pa, ar, pb, br, 0.5j, pc, m)
    torch.cuda.synchronize()
    after = tc_.cpu().numpy()
    assert np.isnan(after[:off]).all() and np.isnan(after[off + 2 * m * n:]).all()
    got = after[off:off + 2 * m * n].reshape(n, m, 2)
    got = (got[..., 0] + 1j * got[..., 1].astype(np.float64)).T
    ref = (0.5 - 0.25j) * (a @ b) + 0.5j * c
    # three products of parts and sums of parts (at most twice as large each), combined
    scale = 0.75 * (np.abs(a.real) + np.abs(a.imag)) @ (np.abs(b.real) + np.abs(b.imag))
    bound = 6 * (INPUT["tf32x3"] + (PER_K["tf32x3"] * k + 4) * 2.0 ** -23) * scale + 2.0 ** -21 * (
        scale + np.abs(c))
    assert (np.abs(got - ref) <= bound).all()
