"""GPU tests of the FP64 split-K forms and of operand copies off a 16-byte
boundary (csrc/dgemm_fp64.cu).

Tile edges, slice counts that are not powers of two, a last slice shorter than
the others, odd leading dimensions (8-byte copies, scalar C) and padding rows
of C; each result against the double-double yardstick of numpy's extended
precision, bar ||C - C_ref||_F <= 8 K u ||A||_F ||B||_F (the parity bar of the
other GEMM tests)."""
import numpy as np
import pytest

from gemm_avx512f_b200 import _lib, blas
from tests._util import fmat, normalized

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("splits", [2, 3, 4, 5, 6, 7, 8, 9])
@pytest.mark.parametrize("tile", [0, 1, 2])
def test_every_slice_count_of_every_tile(cuda, tile, splits):
    import torch

    L = _lib.lib()
    rng = np.random.default_rng(100 * tile + splits)
    # K: `splits` slices of 16 or 32, the last one short; M, N around the tile edges
    for m, n, k, ta, tb, pad, beta in ((64, 64, 16 * splits, "N", "N", 0, 0.0),
                                       (129, 63, 16 * splits - 7, "T", "N", 1, 1.0),
                                       (1, 131, 32 * splits - 31, "N", "T", 3, -0.5),
                                       (200, 66, 32 * splits, "T", "T", 2, 0.5)):
        a = fmat(rng, *((m, k) if ta == "N" else (k, m)), pad=pad)
        b = fmat(rng, *((k, n) if tb == "N" else (n, k)), pad=pad)
        c = fmat(rng, m, n, pad=pad)
        opa = a[:m] if ta == "N" else a[:k].T
        opb = b[:k] if tb == "N" else b[:n].T
        ref = (1.25 * (opa.astype(np.longdouble) @ opb.astype(np.longdouble))
               + beta * c[:m].astype(np.longdouble)).astype(np.float64)
        da, db, dc = (torch.from_numpy(x.T.copy()).to(cuda) for x in (a, b, c))
        torch.cuda.synchronize()
        assert L.b2_set_fp64_config(tile, 8, splits) == 0
        try:
            blas.dgemm_device(ta, tb, m, n, k, 1.25, da, a.shape[0], db, b.shape[0], beta, dc,
                              m + pad)
            torch.cuda.synchronize()
        finally:
            L.b2_set_fp64_config(-1, 0, 0)
        got = dc.cpu().numpy().T
        assert np.array_equal(got[m:], c[m:]), "padding rows of C were written"
        assert normalized(got[:m], ref, k, opa, opb, U) <= 8, (m, n, k, ta, tb)


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("offs", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_operands_off_a_16_byte_boundary(cuda, ta, tb, offs):
    """Bases 8 bytes off and odd / even leading dimensions in every pairing:
    rows are then copied with a shift of one element."""
    import torch

    rng = np.random.default_rng(17)
    for m, n, k, pa, pb in ((129, 130, 77, 0, 1), (64, 128, 64, 1, 1), (257, 65, 160, 2, 3),
                            (63, 64, 5, 1, 0), (1, 2, 1, 0, 0)):
        ar, ac = (m, k) if ta == "N" else (k, m)
        br, bc = (k, n) if tb == "N" else (n, k)
        a, b, c = fmat(rng, ar, ac, pad=pa), fmat(rng, br, bc, pad=pb), fmat(rng, m, n, pad=1)
        opa = a[:ar] if ta == "N" else a[:ar].T
        opb = b[:br] if tb == "N" else b[:br].T
        ref = (opa.astype(np.longdouble) @ opb.astype(np.longdouble)
               + 0.5 * c[:m].astype(np.longdouble)).astype(np.float64)

        def up(x, off):
            # NaN around the operand: a value read from outside would show
            t = torch.full((x.size + 4,), float("nan"), dtype=torch.float64, device=cuda)
            t[off:off + x.size] = torch.from_numpy(x.T.copy().reshape(-1)).to(cuda)
            return t[off:]

        for tile in (0, 1, 2, None):  # None: the call's own choice, 32x32 at these sizes
            da, db, dc = up(a, offs[0]), up(b, offs[1]), up(c, 1)
            torch.cuda.synchronize()
            if tile is not None:
                assert _lib.lib().b2_set_fp64_config(tile, 4, 1) == 0
            try:
                blas.dgemm_device(ta, tb, m, n, k, 1.0, da, a.shape[0], db, b.shape[0], 0.5, dc,
                                  m + 1)
                torch.cuda.synchronize()
            finally:
                _lib.lib().b2_set_fp64_config(-1, 0, 0)
            got = dc[:c.size].cpu().numpy().reshape(n, m + 1).T
            assert np.array_equal(got[m:], c[m:])
            assert normalized(got[:m], ref, k, opa, opb, U) <= 8, (m, n, k, tile)


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
def test_small_tile_edges(cuda, ta, tb):
    """Sizes for which a call takes 32x32 tiles, in one slice and in several:
    around the tile's edges and the K block of 16, long K on one tile, padding."""
    import torch

    rng = np.random.default_rng(29)
    for m, n, k, pad in ((1, 1, 1, 0), (31, 33, 15, 0), (32, 32, 16, 2), (33, 31, 17, 1),
                         (64, 65, 48, 0), (65, 96, 130, 3), (40, 24, 4099, 0), (300, 65, 1000, 0),
                         (130, 1000, 64, 1)):
        a = fmat(rng, *((m, k) if ta == "N" else (k, m)), pad=pad)
        b = fmat(rng, *((k, n) if tb == "N" else (n, k)), pad=pad)
        c = fmat(rng, m, n, pad=pad)
        opa = a[:m] if ta == "N" else a[:k].T
        opb = b[:k] if tb == "N" else b[:n].T
        ref = (1.25 * (opa.astype(np.longdouble) @ opb.astype(np.longdouble))
               - 0.5 * c[:m].astype(np.longdouble)).astype(np.float64)
        da, db, dc = (torch.from_numpy(x.T.copy()).to(cuda) for x in (a, b, c))
        torch.cuda.synchronize()
        blas.dgemm_device(ta, tb, m, n, k, 1.25, da, a.shape[0], db, b.shape[0], -0.5, dc, m + pad)
        torch.cuda.synchronize()
        got = dc.cpu().numpy().T
        assert np.array_equal(got[m:], c[m:]), "padding rows of C were written"
        assert normalized(got[:m], ref, k, opa, opb, U) <= 8, (m, n, k)
