"""GPU tests of the diagonal blocks' inversion (csrc/trsm.cu, trtri_batched_kernel).

Solved against the identity, one block of order <= 128 gives its inverse as it
is stored (products with ones and zeros are exact): every element has to be the
chain of plain substitution, restated here with exactly rounded multiply-adds.
An infinity or a NaN in the triangle reaches the rows that depend on it and no
others."""
from fractions import Fraction

import numpy as np
import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _substitution(T, unit):
    """Inverse of lower triangular T, column by column, k ascending."""
    n = len(T)
    X = np.zeros((n, n))
    inv = [1.0 if unit else 1.0 / T[i, i] for i in range(n)]
    for j in range(n):
        for i in range(j, n):
            acc = 1.0 if i == j else 0.0
            for k in range(j, i):
                acc = _fma(-T[i, k], X[k, j], acc)
            X[i, j] = acc * inv[i]
    return X


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("diag", "NU")
@pytest.mark.parametrize("n", [1, 15, 16, 17, 41])
def test_inverse_is_plain_substitution(cuda, uplo, diag, n):
    import torch

    rng = np.random.default_rng(n)
    low = np.tril(rng.uniform(-1, 1, (n, n)))
    if diag == "U":
        np.fill_diagonal(low, 1.0)
    ref = _substitution(low, diag == "U")
    A = low if uplo == "L" else low[::-1, ::-1]
    ref = ref if uplo == "L" else ref[::-1, ::-1]
    a = torch.from_numpy(A.T.copy()).to(cuda)
    x = torch.eye(n, dtype=torch.float64, device=cuda)
    torch.cuda.synchronize()
    blas.dtrsm_device("L", uplo, "N", diag, n, n, 1.0, a, n, x, n)
    torch.cuda.synchronize()
    assert np.array_equal(x.cpu().numpy().T, ref)


@pytest.mark.parametrize("side", "LR")
@pytest.mark.parametrize("lower,trans", [(True, "N"), (True, "T"), (False, "N"), (False, "T")])
@pytest.mark.parametrize("i,j", [(100, 5), (60, 10), (127, 126), (20, 17), (33, 0)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_elements_stay_in_their_rows(cuda, side, lower, trans, i, j, bad):
    """T = op(A), lower or upper, of order 128 with T(i, j) not finite."""
    import torch

    n, nrhs = 128, 9
    rng = np.random.default_rng(7)
    T = rng.uniform(0.1, 1, (n, n))
    T[np.arange(n), np.arange(n)] += n
    T = np.tril(T)
    T[i, j] = bad
    # the solve's own triangle (side 'R' solves with the transpose)
    if not lower:
        T = T[::-1, ::-1]
        rows = np.arange(n) <= n - 1 - i  # those that depend on the element
        hit = n - 1 - i
    else:
        rows = np.arange(n) >= i
        hit = i
    opA = T if side == "L" else T.T
    uplo = "L" if np.isfinite(np.triu(opA, 1)).all() and not np.triu(opA, 1).any() else "U"
    A = opA if trans == "N" else opA.T
    uplo = uplo if trans == "N" else "UL"[uplo == "U"]
    b = rng.uniform(0.1, 1, (n, nrhs))

    def solve(mat):
        a = torch.from_numpy(np.ascontiguousarray(mat.T)).to(cuda)
        m, k = (n, nrhs) if side == "L" else (nrhs, n)
        x = torch.from_numpy(np.ascontiguousarray((b if side == "L" else b.T).T)).to(cuda)
        torch.cuda.synchronize()
        blas.dtrsm_device(side, uplo, trans, "N", m, k, 1.0, a, n, x, m)
        torch.cuda.synchronize()
        x = x.cpu().numpy().T
        return x if side == "L" else x.T

    got, clean = solve(A), solve(np.where(np.isfinite(A), A, 0.5))
    assert np.array_equal(got[~rows], clean[~rows])
    assert not np.isfinite(got[hit]).any()
    if bad == np.inf and j == 0:  # one element of that row of the inverse is infinite
        assert np.isinf(got[hit]).all()


@pytest.mark.parametrize("row", [0, 40, 127, 200])
@pytest.mark.parametrize("nrhs", [9, 2500])
def test_infinite_right_hand_side(cuda, row, nrhs):
    """An infinity in B stays one in its own row of X, and in its own column."""
    import torch

    n = 256
    rng = np.random.default_rng(row)
    T = np.tril(rng.uniform(0.1, 1, (n, n)))
    T[np.arange(n), np.arange(n)] += n
    b = rng.uniform(0.1, 1, (n, nrhs))

    def solve(rhs):
        a = torch.from_numpy(np.ascontiguousarray(T.T)).to(cuda)
        x = torch.from_numpy(np.ascontiguousarray(rhs.T)).to(cuda)
        torch.cuda.synchronize()
        blas.dtrsm_device("L", "L", "N", "N", n, nrhs, 1.0, a, n, x, n)
        torch.cuda.synchronize()
        return x.cpu().numpy().T

    clean = solve(b)
    for bad in (np.inf, -np.inf, np.nan):
        rhs = b.copy()
        rhs[row, 3] = bad
        got = solve(rhs)
        assert np.array_equal(got[row, 3], bad, equal_nan=True)
        others = np.arange(nrhs) != 3
        assert np.array_equal(got[:, others], clean[:, others])
