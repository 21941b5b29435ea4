"""GPU tests of the small cgemm3m kernel (csrc/gemm3m.cu): tile and K-panel
edges, every transpose pair, padded leading dimensions and operands off an
8-byte boundary, element by element against complex128 products of the same
inputs; surroundings of every operand hold NaN, and C's padding stays as it is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (31, 33, 15), (32, 32, 16), (33, 31, 17), (64, 65, 70), (100, 7, 129),
          (3, 200, 5), (255, 255, 255)]


def _operand(rng, rows, cols, pad, off, dev):
    """A column-major complex64 matrix `off` floats into its buffer."""
    import torch

    ld = rows + pad
    buf = np.full(2 * ld * cols + 8, np.nan, np.float32)
    view = buf[off:off + 2 * ld * cols].reshape(cols, ld, 2)
    view[:, :rows] = rng.uniform(-1, 1, (cols, rows, 2)).astype(np.float32)
    mat = view[:, :rows].astype(np.float64)
    return torch.from_numpy(buf).to(dev), (mat[..., 0] + 1j * mat[..., 1]).T, ld, buf


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("off,pad", [(0, 0), (0, 3), (1, 1)])
def test_small_products(cuda, m, n, k, off, pad):
    import torch

    from gemm_avx512f_b200 import _lib

    lib = _lib.lib()
    rng = np.random.default_rng(m * 1000 + n + k)
    form = {"N": lambda x: x, "T": lambda x: x.T, "R": np.conj, "C": lambda x: x.conj().T}
    st = torch.cuda.Stream()
    for ta in "NTRC":
        for tb in "NTRC":
            a = _operand(rng, *((m, k) if ta in "NR" else (k, m)), pad, off, cuda)
            b = _operand(rng, *((k, n) if tb in "NR" else (n, k)), pad, off, cuda)
            c = _operand(rng, m, n, pad, off, cuda)
            alpha, beta = np.array([1.25, -0.5], np.float32), np.array([0.5, 0.25], np.float32)
            torch.cuda.synchronize()
            assert lib.b2_cgemm3m(
                ta.encode(), tb.encode(), m, n, k, alpha.ctypes.data, a[0].data_ptr() + 4 * off,
                a[2], b[0].data_ptr() + 4 * off, b[2], beta.ctypes.data,
                c[0].data_ptr() + 4 * off, c[2], st.cuda_stream) == 0
            torch.cuda.synchronize()
            al, be = complex(*alpha), complex(*beta)
            oa, ob = form[ta](a[1]), form[tb](b[1])
            ref = al * (oa @ ob) + be * c[1]
            after = c[0].cpu().numpy()
            got = after[off:off + 2 * c[2] * n].reshape(n, c[2], 2)
            assert np.isnan(got[:, m:]).all()
            assert np.isnan(after[:off]).all() and np.isnan(after[off + 2 * c[2] * n:]).all()
            val = (got[:, :m, 0] + 1j * got[:, :m, 1].astype(np.float64)).T
            # each of the three products: k + 1 roundings of sums of at most
            # 2 |a||b| (pre-added operands, one more each); with the post-adds and
            # the complex scaling at most 10 |alpha| |A||B| in magnitude
            u = 2.0 ** -24
            mag = 10 * abs(al) * (np.abs(oa) @ np.abs(ob)) + 4 * abs(be) * np.abs(c[1])
            assert (np.abs(val - ref) <= (k + 8) * u * mag).all(), (ta, tb)
