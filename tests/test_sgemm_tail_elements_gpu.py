"""GPU tests of the FP32 kernel's last partial wave (csrc/sgemm.cu) element by element:
the tiles that run as K slices are a few of all, so a norm over C hardly sees them."""
import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu


def _check(a, b, c0, c, alpha, beta, k):
    """k products and sums in FP32, the scaling and the final add."""
    ref = alpha * (a @ b) + beta * c0
    bound = (k + 4) * 2.0 ** -24 * (abs(alpha) * (a.abs() @ b.abs()) + (beta * c0).abs())
    assert bool(((c - ref).abs() <= bound).all())


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("m,n,k,pad", [
    (3840, 1280, 4096, 0),                   # 300 tiles on 296 slots: 4 in 8 slices
    (128 * 25 - 3, 128 * 12 + 5, 700, 1),    # 325: 29 tiles, 2 slices, 4-byte copies
    (4096, 4096, 512, 4),                    # 1024: 136 tiles in 2 slices
])
def test_last_wave_element_by_element(cuda, ta, tb, m, n, k, pad):
    import torch

    g = torch.Generator(device=cuda).manual_seed(m + n + k)
    ar, ac = (m, k) if ta == "N" else (k, m)
    br, bc = (k, n) if tb == "N" else (n, k)
    mk = lambda r, c: torch.rand(c, r + pad, device=cuda, generator=g) * 2 - 1  # noqa: E731
    A, B, C0 = mk(ar, ac), mk(br, bc), mk(m, n)
    a, b = A[:, :ar].t().double(), B[:, :br].t().double()
    a, b = (a if ta == "N" else a.t()), (b if tb == "N" else b.t())
    C = C0.clone()
    torch.cuda.synchronize()
    blas.sgemm_device(ta, tb, m, n, k, 1.5, A, ar + pad, B, br + pad, -0.5, C, m + pad,
                      method="fp32")
    torch.cuda.synchronize()
    _check(a, b, C0[:, :m].t().double(), C[:, :m].t().double(), 1.5, -0.5, k)
    assert torch.equal(C[:, m:], C0[:, m:]), "padding rows of C were written"


def test_captured_call_of_a_sliced_shape(cuda):
    """The last wave of 4096 x 4096 would run in slices; a captured call holds no scratch
    that a larger call replaces."""
    import torch

    m = n = 4096
    k = 512
    st = torch.cuda.Stream()

    def product(inner):
        a, b = (torch.rand(4096 * inner, device=cuda) for _ in range(2))
        c = torch.zeros(m * n, device=cuda)
        call = lambda: blas.sgemm_device("N", "N", m, n, inner, 1.0, a, m, b, inner, 0.0, c, m,  # noqa: E731
                                         method="fp32", stream=st)
        return a, b, c, call

    a, b, c, call = product(k)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(st):
        with torch.cuda.graph(graph, stream=st):
            call()
    # 1088 tiles: 200 in the last wave, more scratch than the captured shape's
    big = [torch.rand(4352 * 4096, device=cuda) for _ in range(3)]
    torch.cuda.synchronize()
    blas.sgemm_device("N", "N", 4352, 4096, 4096, 1.0, big[0], 4352, big[1], 4096, 0.0, big[2], 4352,
                      method="fp32", stream=st)
    graph.replay()
    torch.cuda.synchronize()
    _check(a.view(k, m).double().t(), b.view(n, k).double().t(),
           torch.zeros(m, n, device=cuda, dtype=torch.float64), c.view(n, m).double().t(), 1.0, 0.0, k)
