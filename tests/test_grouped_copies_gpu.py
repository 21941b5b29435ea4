"""GPU tests of the grouped GEMM's operand copies (csrc/grouped.cu, fp64_copy.cuh,
fp32_copy.cuh): tile and K-block edges, odd and even leading dimensions, bases
off a 16-byte boundary, every transpose pair of both types in one batch, against
FP64 products of the same inputs; surroundings of every operand hold NaN, and
C's padding stays as it is."""
import numpy as np
import pytest

from gemm_avx512f_b200 import _lib

pytestmark = pytest.mark.gpu
SHAPES = [(64, 64, 16), (65, 63, 17), (1, 1, 1), (130, 66, 33), (31, 129, 47), (64, 128, 256),
          (200, 3, 15), (7, 200, 100)]


def test_every_form_in_one_batch(cuda):
    import torch

    rng = np.random.default_rng(12)
    probs, keep = [], []
    for i, (m, n, k) in enumerate(SHAPES):
        for dt in (0, 1):
            for ta in "NT":
                for tb in "NT":
                    for off, pad in ((0, 0), (1, 1), (0, 3), (1, 4), (0, 4)):
                        npdt = (np.float64, np.float32)[dt]
                        ar, ac = (m, k) if ta == "N" else (k, m)
                        br, bc = (k, n) if tb == "N" else (n, k)
                        ops = []
                        for r, c in ((ar, ac), (br, bc), (m, n)):
                            ld = r + pad
                            buf = np.full(ld * c + 8, np.nan, npdt)
                            mat = rng.uniform(-1, 1, (c, r)).astype(npdt)
                            view = buf[off:off + ld * c].reshape(c, ld)
                            view[:, :r] = mat
                            ops.append((torch.from_numpy(buf).to(cuda), mat.T, ld, buf))
                        es = npdt().itemsize
                        beta = (0.0, 1.0, -0.5)[i % 3]
                        probs.append(_lib.GemmProblem(
                            dt, ta.encode(), tb.encode(), m, n, k, 1.25, beta,
                            ops[0][0].data_ptr() + off * es, ops[0][2],
                            ops[1][0].data_ptr() + off * es, ops[1][2],
                            ops[2][0].data_ptr() + off * es, ops[2][2]))
                        keep.append((dt, ta, tb, m, n, k, beta, off, ops))
    torch.cuda.synchronize()
    arr = (_lib.GemmProblem * len(probs))(*probs)
    st = torch.cuda.Stream()
    assert _lib.lib().b2_gemm_grouped(len(arr), arr, st.cuda_stream) == 0
    torch.cuda.synchronize()
    for dt, ta, tb, m, n, k, beta, off, ops in keep:
        a, b, c = (x[1].astype(np.float64) for x in ops)
        a, b = (a if ta == "N" else a.T), (b if tb == "N" else b.T)
        ref = 1.25 * (a @ b) + beta * c
        ld, before = ops[2][2], ops[2][3]
        after = ops[2][0].cpu().numpy()
        got = after[off:off + ld * n].reshape(n, ld)
        assert np.isnan(got[:, m:]).all() and np.isnan(after[off + ld * n:]).all()
        assert np.array_equal(np.isnan(before[:off]), np.isnan(after[:off]))
        u = (2.0 ** -53, 2.0 ** -24)[dt]
        err = np.linalg.norm(got[:, :m].T - ref)
        bar = 8 * max(k, 1) * u * 1.25 * np.linalg.norm(a) * np.linalg.norm(b) + 4 * u * np.linalg.norm(ref)
        assert err <= bar, (dt, ta, tb, m, n, k, off, ld, err, bar)
