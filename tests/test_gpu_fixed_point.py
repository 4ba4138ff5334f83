"""FP64 sums in fixed point (csrc/fx.cuh): bricks whose values allow it are summed in integers, the
others in FP64, and both kinds sit side by side in one sweep.  Checked against the oracle's FP64
array sweep at values that reach every branch: all bricks in integers, values that are zero in part,
magnitudes that force some or all bricks to FP64, infinities and NaNs, the largest and the smallest
doubles, brick lists of one and of an odd number, output fields off the 16-byte boundary.

Tolerance, point by point: both sides sum n products; the oracle rounds each product and sum
(2n roundings), and the kernel's error is bounded by n roundings of its largest term, so
|got - want| <= 3 n 2^-53 sum |c x|.
"""
import numpy as np
import pytest

from bricklib_gb300 import bricks as B, stencils
from bricklib_gb300._abi import BK_F64
from bricklib_gb300.domain import GridDomain
from oracle import oracle

pytestmark = pytest.mark.gpu

CUBE = stencils.cube_taps(1)[0]


def stencil(name):
    if name == "star25-uneven":  # 25 different coefficients: one product per tap
        taps, _ = stencils.star_taps(4)
        return stencils.custom(name, taps, stencils.uniform(3, len(taps), 0.5, 1.0))
    if name == "star13-uneven":
        taps, _ = stencils.star_taps(2)
        return stencils.custom(name, taps, stencils.uniform(4, len(taps), -1.0, -0.5))
    if name == "cube27-signs":
        return stencils.custom(name, CUBE, stencils.uniform(5, 27, 0.5, 1.0) * np.where(np.arange(27) % 3 == 1, -1, 1))
    return stencils.make(name, 5)


STENCILS = ["star7", "heat7", "star13", "star25", "star13-uneven", "star25-uneven", "cube27", "cube27-signs", "cube125"]


def values(kind, dims, org):
    a = stencils.uniform(77, int(np.prod(dims))).reshape(dims)
    rng = np.random.default_rng(1)
    if kind == "zeros":  # zero but for a few cells: integers where every value is exact
        a = np.where(rng.random(dims) < 0.002, np.round(a, 1), 0.0)
    elif kind == "spread":  # thirty binary orders of magnitude from cell to cell
        a = a * 2.0 ** rng.integers(-30, 1, dims)
    elif kind == "decay":  # falls by 2^2 per cell along i, from 1
        a = a * 2.0 ** (-2.0 * np.arange(dims[2]))
    elif kind == "huge":
        a = a * 1e300
    elif kind == "tiny":  # around the smallest normal number: products underflow
        a = a * 1e-306
    elif kind == "inf":
        a[org[0] + 9, org[1] + 3, org[2] + 4] = np.inf
        a[org[0] + 9, org[1] + 20, org[2] + 30] = np.nan
        a[org[0] + 20, org[1] + 7, org[2] + 8] = -np.inf
    return np.ascontiguousarray(a)


def check(dom, arr, st, got):
    o, n = dom.org, dom.n
    want, size = np.zeros_like(arr), np.zeros_like(arr)
    end = tuple(a + b for a, b in zip(o, n))
    with np.errstate(all="ignore"):
        oracle.array_sweep(arr, want, o, end, st.offsets(), st.coeff)
        oracle.array_sweep(np.abs(arr), size, o, end, st.offsets(), np.abs(st.coeff))
        want, size = dom.interior_view(want), dom.interior_view(size)
        fine = np.isfinite(want)
        assert np.array_equal(fine, np.isfinite(got))
        assert np.array_equal(np.isnan(want), np.isnan(got))
        assert np.array_equal(want[np.isinf(want)], got[np.isinf(want)])
        # products and sums below the smallest normal number round to multiples of 2^-1074
        bound = 3 * st.npoints * (2.0 ** -53 * size[fine] + 2.0 ** -1074)
        bad = np.abs(got[fine] - want[fine]) > bound
    assert not bad.any(), (int(bad.sum()), float(np.max(np.abs(got[fine] - want[fine]) / np.maximum(size[fine], 1e-320))))


@pytest.mark.parametrize("kind", ["uniform", "zeros", "spread", "decay", "huge", "tiny", "inf"])
@pytest.mark.parametrize("name", STENCILS)
def test_fixed_point_sweeps_against_the_oracle(name, kind):
    st = stencil(name)
    dom = GridDomain((24, 32, 40), dtype=BK_F64)
    arr = values(kind, dom.adims, dom.org)
    dom.set_field(0, arr)
    dom.upload()
    B.brickSweep(dom.brick(0), dom.brick(1), dom.dev_interior, st)
    B.synchronize()
    assert B.error_flags() == 0
    dom.download()
    check(dom, arr, st, dom.interior_view(dom.get_field(1)))


@pytest.mark.parametrize("name", STENCILS)
def test_fixed_point_zero_bricks(name):
    """Bricks whose values are all zero (of either sign) are not summed; denormals beside zeros are."""
    st = stencil(name)
    dom = GridDomain((24, 32, 40), dtype=BK_F64)
    arr, o = np.zeros(dom.adims), dom.org
    arr[o[0]:o[0] + 8, o[1]:o[1] + 12] = -0.0
    arr[o[0] + 16:o[0] + 24, o[1] + 8:o[1] + 16, o[2] + 8:o[2] + 16] = 1e-320
    arr[o[0] + 8, o[1] + 24, o[2] + 24] = 1e-318  # a corner of one brick, in the reach of its neighbours
    arr[o[0] + 12:o[0] + 14, o[1] + 3, o[2] + 30:] = 0.75
    dom.set_field(0, arr)
    dom.upload()
    B.brickSweep(dom.brick(0), dom.brick(1), dom.dev_interior, st)
    B.synchronize()
    assert B.error_flags() == 0
    dom.download()
    check(dom, arr, st, dom.interior_view(dom.get_field(1)))


@pytest.mark.parametrize("name", ["star7", "star13", "star25", "cube27", "cube125"])
@pytest.mark.parametrize("count,off", [(1, 0), (7, 0), (60, 1)])
def test_fixed_point_short_lists_and_odd_output_fields(name, count, off):
    """One brick, an odd number of them, and an output field whose bricks start at odd elements:
    the listed bricks equal the full sweep's (the oracle's, where another kernel stores them)."""
    st = stencil(name)
    dom = GridDomain((24, 32, 40), dtype=BK_F64)
    arr = values("uniform", dom.adims, dom.org)
    dom.set_field(0, arr)
    dom.upload()
    B.brickSweep(dom.brick(0), dom.brick(1), dom.dev_interior, st)
    ids = dom.interior[:count]
    step = 512 + 2 * off
    ost = B.BrickStorage.allocate_device(dom.nbricks, step + off, BK_F64)
    B.brickSweep(dom.brick(0), B.Brick(dom.dev_info, ost, off, dom.layout), B.BrickList(ids), st)
    B.synchronize()
    assert B.error_flags() == 0
    dom.download()
    check(dom, arr, st, dom.interior_view(dom.get_field(1)))
    full = dom.storage.host.reshape(dom.nbricks, 2, 512)[:, 1]
    got = B.movBrickStorage(ost, to_device=False).host.reshape(dom.nbricks, -1)[:, off:off + 512]
    np.testing.assert_allclose(got[ids], full[ids], rtol=0, atol=3 * st.npoints * 2.0 ** -53 * float(np.abs(st.coeff).sum()))
    others = np.setdiff1d(np.arange(dom.nbricks), ids)
    assert not got[others].any()


@pytest.mark.parametrize("kind", ["uniform", "same", "spread", "huge", "inf"])
@pytest.mark.parametrize("ring", [True, False])
def test_fixed_point_4d_stars_against_plain_sums(ring, kind):
    """The radius-1 star on 4-D bricks: one coefficient for the eight neighbours (the values are
    added before they are multiplied; `same`: all values just below a power of two, whose sum is the
    largest there is), and nine different ones."""
    from bricklib_gb300 import bricks4 as B4
    lay, g = B4.Layout4(), (4, 3, 5, 4)
    grid, adj = B4.init_grid(list(reversed(g)))
    dims = tuple(4 * x for x in g)
    arr = stencils.uniform(5, int(np.prod(dims))).reshape(dims)
    rng = np.random.default_rng(2)
    if kind == "same":
        arr = np.full(dims, 1.0 - 2.0 ** -53)
    elif kind == "spread":
        arr = arr * 2.0 ** rng.integers(-40, 1, dims)
    elif kind == "huge":
        arr = arr * 1e299
    elif kind == "inf":
        arr[5, 5, 6, 7] = np.inf
        arr[9, 6, 9, 5] = np.nan
    st = B4.mpi9pt()
    if not ring:
        st.coeff = stencils.uniform(8, 9, 0.5, 1.0)
    host = np.zeros(len(grid) * 512)
    B4.copy_to_bricks(arr, grid, g, (0, 0, 0, 0), host, 512, 0, lay)
    dev = B.movBrickStorage(B.BrickStorage(len(grid), 512, BK_F64, host=host))
    a = B.DeviceBuffer(adj.nbytes)
    a.upload(adj)
    inner = grid.reshape(g)[1:-1, 1:-1, 1:-1, 1:-1]
    B4.sweep4(a, len(grid), dev, 0, 256, B.BrickList(np.ascontiguousarray(inner.reshape(-1))), st, lay)
    B.synchronize()
    assert B.error_flags() == 0
    out = B.movBrickStorage(dev, to_device=False).host
    ig = tuple(x - 2 for x in g)
    got = np.zeros(tuple(4 * x for x in ig))
    B4.copy_from_bricks(got, inner, ig, (0, 0, 0, 0), out, 512, 256, lay)
    want, size = np.zeros_like(got), np.zeros_like(got)
    with np.errstate(all="ignore"):
        for tap, c in zip(st.taps, st.coeff):
            v = arr[tuple(slice(4 + o, 4 + o + n) for o, n in zip(tap, got.shape))]
            want = want + c * v
            size = size + np.abs(c * v)
        fine = np.isfinite(want)
        assert np.array_equal(fine, np.isfinite(got)) and np.array_equal(np.isnan(want), np.isnan(got))
        assert (np.abs(got[fine] - want[fine]) <= 3 * 9 * 2.0 ** -53 * size[fine]).all()
