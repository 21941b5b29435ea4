"""GPU test of cgemm3m where the device has no room for the scratch of its batched form
(csrc/sgemm_tc.cu): the three products then run one after another in less than the
former three-GEMM form took."""
import threading

import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(6000, 6000, 6000), (3000, 2000, 30000)])
def test_products_one_after_another(cuda, m, n, k):
    import torch

    g = torch.Generator(device=cuda).manual_seed(m)
    rnd = lambda cnt: torch.view_as_complex(  # noqa: E731
        torch.rand(cnt, 2, device=cuda, generator=g) * 2 - 1)
    a, b, c0 = rnd(m * k), rnd(k * n), rnd(m * n)
    results, errors = [c0.clone(), c0.clone()], []
    torch.cuda.synchronize()

    def call(c):
        try:
            blas.cgemm3m_device("N", "N", m, n, k, 0.5 - 1j, a, m, b, k, 0.25j, c, m)
            torch.cuda.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    def in_thread(c):  # of its own: a context without scratch from earlier calls
        t = threading.Thread(target=call, args=(c,))
        t.start()
        t.join()

    call(results[0])  # (in this thread: its context keeps its scratch)
    # what the three-GEMM form took: 3 (m k + k n + m n) floats of parts, 2 (m + n) k of
    # segments; the batched form takes 6 (m + n) k and its sums
    former = 4 * (3 * (m * k + k * n + m * n) + 2 * (m + n) * k)
    spare = 64 << 20  # the context's small buffers
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    fill = torch.empty(max(0, free - former - spare), dtype=torch.uint8, device=cuda)
    try:
        in_thread(results[1])
    finally:
        del fill
        torch.cuda.empty_cache()
    assert not errors, errors
    prod = b.view(n, k).to(torch.complex128) @ a.view(k, m).to(torch.complex128)
    ref = (0.5 - 1j) * prod + 0.25j * c0.view(n, m).to(torch.complex128)
    for got in results:
        err = float((got.view(n, m) - ref).norm() / ref.norm())
        assert err <= 2e-6 + 2e-8 * k, err  # the 3xTF32 bar of the SGEMM tests
