"""GPU tests of how the tensor-core SGEMM forms accumulate K (csrc/sgemm_tc.cu,
csrc/umma.cuh): the ranges of a split are chains of their own, down to one term of
one K block, on every engine.

The inputs make the place of a range's end visible exactly: a chain that held the
large term together with the 1 that follows it would drop the 1 (2^27 + 4097 is not
an FP32 number) before the large term is taken away again."""
import numpy as np
import pytest

from gemm_avx512f_b200 import _lib

pytestmark = pytest.mark.gpu
METHOD = {"tf32": 0, "tf32x3": 1, "bf16x3": 2}  # of b2_sgemm_config
KBLOCK = {"tf32": 32, "tf32x3": 32, "bf16x3": 64}


def _run(cuda, method, engine, log2split, a, b):
    """a (m x k) times b (k x n) with a given engine and split."""
    import torch

    m, k = a.shape
    n = b.shape[1]
    da = torch.from_numpy(np.ascontiguousarray(a.T)).to(cuda)
    db = torch.from_numpy(np.ascontiguousarray(b.T)).to(cuda)
    dc = torch.zeros((n, m), device=cuda)
    torch.cuda.synchronize()
    assert _lib.lib().b2_sgemm_config(b"N", b"N", m, n, k, 1.0, da.data_ptr(), m, db.data_ptr(), k,
                                      0.0, dc.data_ptr(), m,
                                      METHOD[method] * 16 + engine * 4 + log2split, None) == 0
    torch.cuda.synchronize()
    return dc.cpu().numpy().T


@pytest.mark.parametrize("engine", [0, 1, 2])
@pytest.mark.parametrize("method", ["tf32x3", "bf16x3"])
@pytest.mark.parametrize("m,n", [(1, 1), (130, 70), (256, 300)])
def test_terms_of_a_k_block_are_chains_of_their_own(cuda, method, engine, m, n):
    """Two K blocks in 8 ranges: six, one per term."""
    kb = KBLOCK[method]
    s = 4096.0 if method == "tf32x3" else 256.0  # s + 1 needs one bit more than a segment holds
    big = 2.0 ** 27 / s
    a, b = np.zeros((m, 2 * kb), np.float32), np.zeros((2 * kb, n), np.float32)
    a[:, [0, 1, kb, kb + 1]] = [big, 1.0, -big, -1.0]
    b[[0, 1, kb, kb + 1]] = np.array([[s], [s + 1], [s], [s]], np.float32)
    assert (_run(cuda, method, engine, 3, a, b) == 1.0).all()


def _in_k_blocks(method, m, n, values):
    """Operands whose K block i holds the one product values[i][0] * values[i][1]."""
    kb = KBLOCK[method]
    a = np.zeros((m, len(values) * kb), np.float32)
    b = np.zeros((len(values) * kb, n), np.float32)
    a[:, ::kb] = [x for x, _ in values]
    b[::kb] = np.array([[y] for _, y in values], np.float32)
    return a, b


@pytest.mark.parametrize("engine", [0, 1, 2])
@pytest.mark.parametrize("method", sorted(METHOD))
@pytest.mark.parametrize("log2split", [2, 3])
@pytest.mark.parametrize("m,n", [(128, 100), (1024, 1024), (2300, 1500)])
def test_ranges_are_added_as_in_fp64(cuda, method, engine, log2split, m, n):
    """Eight K blocks in 4 or 8 ranges, one unit per tile (many tiles) or several: the
    ranges' sums are added with their rounding errors (eight bits of them, where one
    unit adds several ranges) and rounded once."""
    zero = (0.0, 0.0)

    def run(first, second, third):
        # two K blocks apart: different ranges of four as well
        v = [first, zero, second, zero, third, zero, zero, zero]
        return _run(cuda, method, engine, log2split, *_in_k_blocks(method, m, n, v))

    # FP32 additions in order would drop the 1
    assert (run((2.0 ** 14, 2.0 ** 13), (1.0, 1.0), (-2.0 ** 14, 2.0 ** 13)) == 1.0).all()
    # ... and the last bit here: 2^24 + 1 + 2^-6 lies above the middle of two floats
    assert (run((2.0 ** 12, 2.0 ** 12), (1.0, 1.0), (2.0 ** -3, 2.0 ** -3)) == 2.0 ** 24 + 2).all()
    # ... and pass FLT_MAX on the way to a sum that does not
    x = (2.0 ** 64, 1.5 * 2.0 ** 63)
    assert (run(x, x, (-x[0], x[1])) == np.float32(1.5 * 2.0 ** 127)).all()
    assert np.isposinf(run(x, x, zero)).all()
    if method == "tf32":  # (the split forms make a NaN of an infinite operand's small part)
        assert np.isposinf(run((np.inf, 1.0), (1.0, 1.0), (-1.0, 2.0))).all()
        assert np.isnan(run((np.inf, 1.0), (1.0, 1.0), (-np.inf, 1.0))).all()
