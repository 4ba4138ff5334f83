"""The host's side of the FP64 sums in fixed point (csrc/fx.cuh, fx_table): which stencils are
summed in integers, and what the device's check of a brick lets through.  No GPU: the table is made
by the library's own function and its rule is restated here in exact numbers."""
import ctypes as C
import struct
from fractions import Fraction

import pytest

from bricklib_gb300 import _abi, stencils

TAPS = 27


class Table(C.Structure):
    _fields_ = [("on", C.c_int), ("ch", C.c_int * TAPS), ("cl", C.c_int * TAPS), ("w", C.c_int * 8),
                ("elo", C.c_int), ("ehi", C.c_int), ("q", C.c_int), ("zeros", C.c_int)]


def tap_list(kind, r):
    """Kernel order: star: the centre, then the rings; cube: row-major."""
    if kind == "cube":
        return [(k, j, i) for k in range(-r, r + 1) for j in range(-r, r + 1) for i in range(-r, r + 1)]
    out = [(0, 0, 0)]
    for d in range(1, r + 1):
        out += [(0, 0, d), (0, 0, -d), (0, d, 0), (0, -d, 0), (d, 0, 0), (-d, 0, 0)]
    return out


def table(kind, r, coeff):
    """fx_table with one product per tap; (usable, the table)."""
    taps = tap_list(kind, r)
    n = len(taps)
    masks = 8 if kind == "cube" else 5
    near = ((C.c_int * 9) * 8)()
    for m in range(8):
        at = [t for t, tap in enumerate(taps)
              if tuple(abs(x) for x in tap) == (m >> 2 & 1, m >> 1 & 1, m & 1)]
        if kind == "star" and m & (m - 1):
            at = [0]
        near[m][:len(at) + 1] = at + [-1]
    f = _abi.lib()._ZN2bk8fx_tableEPKdiPA9_KiiiPS2_S5_ibPNS_5FxTabE
    f.restype = C.c_bool
    first, count, t = (C.c_int * n)(*range(n)), (C.c_int * n)(*[1] * n), Table()
    ok = f((C.c_double * n)(*coeff), n, near, masks, n, first, count, 60, C.c_bool(kind == "star" and r == 1), C.byref(t))
    return bool(ok), t


def test_table_of_ordinary_stencils():
    for kind, r in (("star", 1), ("star", 2), ("cube", 1)):
        n = len(tap_list(kind, r))
        ok, t = table(kind, r, stencils.uniform(9, n, 0.5, 1.0))
        assert ok and t.elo < 1023 < t.ehi, (kind, r)


@pytest.mark.parametrize("kind,r", [("star", 1), ("star", 2), ("star", 4), ("cube", 1)])
def test_power_of_two_neighbours_stay_in_fp64_whatever_the_centre(kind, r):
    """Coefficients that are powers of two but for the centre's (Laplacians): the products of the
    neighbours are exact in FP64, which such stencils keep.  Another tap's coefficient takes that
    away, wherever in the kernel's order it stands."""
    taps = tap_list(kind, r)
    centre = taps.index((0, 0, 0))
    powers = [0.5] * len(taps)
    powers[centre] = -5.7
    assert not table(kind, r, powers)[0]
    for other in {0, 1, centre - 1, len(taps) - 1} - {centre, -1}:
        uneven = [0.5] * len(taps)
        uneven[other] = 0.7
        assert table(kind, r, uneven)[0], other


def high(x):
    """High word of a double, without its sign (the device's fx_mag)."""
    return struct.unpack("<q", struct.pack("<d", x))[0] >> 32 & 0x7FFFFFFF


def double_of(word):
    return struct.unpack("<d", struct.pack("<q", word << 32))[0]


@pytest.mark.parametrize("kind,r", [("star", 1), ("star", 2), ("cube", 1)])
def test_accepted_terms_cover_the_error_they_are_checked_for(kind, r):
    """A brick of largest exponent E is accepted where a checked term c x of every point has
    high(x) + w >= E as high words.  The smallest x that passes must still have
    |c x| n 2^-53 >= the error bound of the sum in integers (units of 2^(E - 1022)): values cut below
    2^-60, coefficients rounded to 2^-q, the roundings to 2^64, and the products cl xl left out."""
    taps = tap_list(kind, r)
    n, E = len(taps), 1023
    for seed in range(200):
        coeff = stencils.uniform(seed, n, 0.5, 1.0)
        ok, t = table(kind, r, coeff)
        if not ok:
            continue
        q = int(t.q)
        one = kind == "star" and r == 1
        error = (sum(Fraction(c) for c in coeff) * Fraction(1, 2 ** 60) + Fraction(n, 2) / 2 ** q +
                 Fraction(1 if one else 2, 2) * Fraction(2) ** (64 - q - 60) +
                 sum(abs(int(x)) for x in t.cl[:n]) * Fraction(2) ** (31 - q - 60))
        unit = Fraction(2) ** (E - 1022)
        for m in range(8 if kind == "cube" else 5):
            at = [k for k, tap in enumerate(taps) if tuple(abs(x) for x in tap) == (m >> 2 & 1, m >> 1 & 1, m & 1)]
            if not at:
                continue
            x = double_of((E << 20) - int(t.w[m]))  # the smallest that passes
            assert high(x) + t.w[m] >= E << 20 > high(x) - 1 + t.w[m]
            term = min(Fraction(float(coeff[k])) for k in at) * Fraction(x)
            assert term * n / 2 ** 53 >= error * unit, (seed, m, float(term * n / 2 ** 53 / (error * unit)))
