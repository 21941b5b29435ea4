"""CPU check of the shifted-row copies of csrc/dgemm_fp64.cu (operands whose
base or leading dimension is odd): every copy is 16-byte aligned (8-byte for
the operand's first element), inside the operand, and every element a fragment
reads is where the fragment looks for it, zero beyond the matrix."""
import pytest

BK, NT = 16, 128


def _copy_pair(mem, sm, dst, base, ld, row, rows, e0, lim, sh):
    valid = max(0, min(2, lim - e0)) if row < rows else 0
    if sh and e0 < 0 and row == 0:
        sm[dst + 1] = mem[base] if valid > 1 else 0
        return
    if valid:
        assert (base + row * ld + e0) % 2 == 0, "misaligned 16-byte copy"
    for j in range(2):
        sm[dst + j] = mem[base + row * ld + e0 + j] if j < valid else 0


def _stage(mem, base, ld, kcont, outer, o0, k0, olim, klim, kbeg, kt):
    """Shared image of one stage (the kernel's load_stage for one operand)."""
    rows, length = (outer, BK) if kcont else (BK, outer)
    pitch = length + 4
    sm = [None] * (rows * pitch)
    r0, c0 = (o0, k0) if kcont else (k0, o0)
    rlim, clim = (olim, klim) if kcont else (klim, olim)
    first = (o0 if kcont else kbeg) == 0
    run = k0 + BK <= klim and not (kt == 0 and first)  # from running pointers
    inside = run and o0 + outer <= olim
    cpr = length // 2
    for tid in range(NT):
        sh = (base + (r0 + tid // cpr) * ld) & 1
        for i in range(outer * BK // 2 // NT):
            c = tid + i * NT
            hi, lo = c // cpr, (c % cpr) * 2
            assert sh == (base + (r0 + hi) * ld) & 1, "the shift is a constant of the thread"
            if inside:
                a = base + (r0 + hi) * ld + c0 + lo - sh
                assert a % 2 == 0 and a >= base
                for j in range(2):
                    sm[hi * pitch + lo + j] = mem[a + j]
            elif run:  # past the outer limit: edge_bytes
                if kcont:
                    valid = 2 if i * (NT // cpr) < olim - o0 - tid // cpr else 0
                else:
                    valid = max(0, min(2, olim - (o0 + (tid % cpr) * 2 - sh)))
                a = base + (r0 + hi) * ld + c0 + lo - sh
                if valid:
                    assert a % 2 == 0 and a >= base
                for j in range(2):
                    sm[hi * pitch + lo + j] = mem[a + j] if j < valid else 0
            else:
                _copy_pair(mem, sm, hi * pitch + lo, base, ld, r0 + hi, rlim, c0 + lo - sh, clim,
                           True)
    for tid in range(rows):
        if (base + (r0 + tid) * ld) & 1:
            _copy_pair(mem, sm, tid * pitch + length, base, ld, r0 + tid, rlim, c0 + length - 1,
                       clim, True)
    return sm, pitch, r0, c0


class _Mem(dict):
    def __missing__(self, key):
        raise AssertionError(f"read outside the operand: element {key}")


@pytest.mark.parametrize("kcont", [True, False])
@pytest.mark.parametrize("base", [0, 1])
@pytest.mark.parametrize("outer", [64, 32])
@pytest.mark.parametrize("outer_n,kn,pad", [(64, 16, 1), (65, 33, 0), (130, 47, 1), (63, 15, 2),
                                            (129, 32, 0), (1, 1, 0)])
def test_shifted_rows_hold_what_the_fragments_read(kcont, base, outer, outer_n, kn, pad):
    ld = (kn if kcont else outer_n) + pad
    nrows = outer_n if kcont else kn
    last = base + (nrows - 1) * ld + (kn if kcont else outer_n)
    mem = _Mem({a: a + 1 for a in range(base, last)})  # only the operand itself
    chunk = 32
    for kbeg in range(0, kn, chunk):
        kend = min(kn, kbeg + chunk)
        for o0 in range(0, outer_n, outer):
            for kt in range((kend - kbeg + BK - 1) // BK):
                k0 = kbeg + kt * BK
                sm, pitch, r0, c0 = _stage(mem, base, ld, kcont, outer, o0, k0, outer_n, kend,
                                           kbeg, kt)
                for o in range(outer):
                    for k in range(BK):
                        # the fragment's shift comes from g or t: row index mod 2
                        r, c = (o, k) if kcont else (k, o)
                        fs = (base + r * ld) & 1
                        got = sm[r * pitch + c + fs]
                        go, gk = o0 + o, k0 + k
                        want = 0
                        if go < outer_n and gk < kend:
                            want = base + (go * ld + gk if kcont else gk * ld + go) + 1
                        assert got == want, (o, k, got, want)
