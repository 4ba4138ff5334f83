"""Which arithmetic an FP64 brick gets, and that it is what it is said to be: fixed point (csrc/fx.cuh)
on uniform values, shown by an error that the FP64 chain does not reach; FP64, bit for bit, where a
brick is refused; the sign of zero sums.  Exact sums and fused multiply-adds are made on the host."""
from fractions import Fraction

import numpy as np
import pytest

from bricklib_gb300 import bricks as B, stencils
from bricklib_gb300._abi import BK_ACC_NATIVE, BK_F64
from bricklib_gb300.domain import GridDomain
from oracle import oracle
from test_gpu_fixed_point import stencil
from test_gpu_sweep import _sweep_with

pytestmark = pytest.mark.gpu

KERNELS = (None, "BK_SWEEP_PIPELINED", "BK_SWEEP_ONESHOT")


def wide(dims, seed=1):
    """Four hundred binary orders of magnitude from cell to cell: the check refuses every brick."""
    rng = np.random.default_rng(seed)
    return stencils.uniform(77, int(np.prod(dims))).reshape(dims) * 2.0 ** rng.integers(-200, 201, dims)


def domain(n=(24, 32, 40)):
    return GridDomain(n, dtype=BK_F64)


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def interior(dom, out):
    dom.storage.host.reshape(dom.nbricks, dom.nfields, -1)[:, 1, :] = \
        out.reshape(dom.nbricks, dom.nfields, -1)[:, 1, :]
    return dom.interior_view(dom.get_field(1))


def points(dom, count, seed=3):
    rng = np.random.default_rng(seed)
    return np.stack([rng.integers(0, m, count) for m in dom.n], axis=1)


@pytest.mark.parametrize("name", ["star7", "star13", "star25", "heat7", "star13-uneven", "star25-uneven"])
def test_refused_star_bricks_are_the_fp64_chain(name, monkeypatch):
    """Stars on values that refuse every brick: the three star kernels give the same bits, those of
    n fused multiply-adds from the centre outwards, ring by ring (+i, -i, +j, -j, +k, -k)."""
    st = stencil(name)
    dom = domain()
    arr = wide(dom.adims)
    dom.set_field(0, arr)
    dom.upload()
    got = [_sweep_with(env, monkeypatch, dom, st, BK_ACC_NATIVE, dom.dev_interior) for env in KERNELS]
    for other in got[1:]:
        np.testing.assert_array_equal(got[0].view(np.uint8), other.view(np.uint8))
    out = interior(dom, got[0])
    coeff = dict(zip([tuple(t) for t in st.taps], [float(c) for c in st.coeff]))
    order = [(0, 0, 0)]
    for d in range(1, st.radius + 1):
        order += [(0, 0, d), (0, 0, -d), (0, d, 0), (0, -d, 0), (d, 0, 0), (-d, 0, 0)]
    o = dom.org
    for p in points(dom, 1500):
        v = 0.0
        for t in order:
            v = fma(coeff[t], float(arr[tuple(o[a] + p[a] + t[a] for a in range(3))]), v)
        assert out[tuple(p)] == v, (p, out[tuple(p)], v)


def plane_sum(coeff, x):
    """The 125-point cube at one point as a refused brick sums it, x[5][5][5] its values: plane by
    plane rows added pairwise, the six class sums of the plane, their weighted sum for the plane's
    distance along k; the planes' sums added from the lowest to the highest."""
    total = None
    for k in range(5):
        V = [x[k, 2], x[k, 1] + x[k, 3], x[k, 0] + x[k, 4]]

        def two(b, a):
            return V[b][2 - a] + V[b][2 + a]

        q = [V[0][2], two(0, 1) + V[1][2], two(1, 1), two(0, 2) + V[2][2], two(1, 2) + two(2, 1), two(2, 2)]
        d, w = abs(k - 2), 0.0
        for c, v in zip([(0, 0), (0, 1), (1, 1), (0, 2), (1, 2), (2, 2)], q):
            w = fma(coeff[(d,) + c], float(v), w)
        total = w if total is None else total + w
    return total


@pytest.mark.parametrize("part", [1.0, 0.5])
def test_refused_cube125_bricks_are_summed_in_fp64(part, monkeypatch):
    """The 125-point cube on values that refuse every brick, or about half of them in stretches of
    one to three, with bricks of zeros between: a refused brick's bits are those of the FP64 sums
    plane by plane, and no brick's depend on what the list has around it."""
    st = stencil("cube125")
    dom = domain((24, 32, 128))
    rng = np.random.default_rng(5)
    arr = wide(dom.adims)
    if part < 1:
        plain = stencils.uniform(78, arr.size).reshape(arr.shape)
        calm = rng.random([m // 8 for m in arr.shape]) >= 0.02
        arr = np.where(np.repeat(np.repeat(np.repeat(calm, 8, 0), 8, 1), 8, 2), plain, arr)
    arr[dom.org[0]:, :, dom.org[2] + 40:dom.org[2] + 60] = 0.0  # bricks of zeros
    dom.set_field(0, arr)
    dom.upload()
    it = np.asarray(dom.interior, dtype=np.uint32)
    cuts = np.cumsum(rng.integers(1, 6, size=len(it)))
    pieces = np.split(it, cuts[cuts < len(it)])
    lists = {"grid": it, "shuffled": rng.permutation(it),
             "pieces": np.concatenate([pieces[p] for p in rng.permutation(len(pieces))]),
             "repeats": np.repeat(it, rng.integers(1, 3, size=len(it)))}
    full = None
    for key, lst in lists.items():
        got = _sweep_with(None, monkeypatch, dom, st, BK_ACC_NATIVE, B.BrickList(np.ascontiguousarray(lst)))
        full = got if full is None else full
        np.testing.assert_array_equal(got.view(np.uint8), full.view(np.uint8), err_msg=key)
    out = interior(dom, full)
    coeff = {t: float(c) for t, c in zip([tuple(t) for t in st.taps], st.coeff)}
    o, same = dom.org, 0
    pts = points(dom, 600)
    for p in pts:
        x = arr[tuple(slice(o[a] + p[a] - 2, o[a] + p[a] + 3) for a in range(3))]
        same += out[tuple(p)] == plane_sum(coeff, x)
    # every point of a refused brick; of the accepted ones only those whose two roundings agree
    assert same == len(pts) if part == 1 else 0.2 * len(pts) < same < 0.95 * len(pts), same
    want = np.zeros_like(arr)
    oracle.array_sweep(arr, want, o, tuple(a + b for a, b in zip(o, dom.n)), st.offsets(), st.coeff)
    size = np.zeros_like(arr)
    oracle.array_sweep(np.abs(arr), size, o, tuple(a + b for a, b in zip(o, dom.n)), st.offsets(), np.abs(st.coeff))
    assert (np.abs(out - dom.interior_view(want)) <= 3 * 125 * 2.0 ** -53 * dom.interior_view(size)).all()


@pytest.mark.parametrize("name", ["star7", "heat7", "star13", "star25", "cube27", "cube125"])
def test_uniform_values_are_summed_in_fixed_point(name):
    """On uniform values the error is that of one rounding to a double: a rounding is uniform in
    half a unit of the last place either way, rms ulp / sqrt(12), and what the sum in integers adds
    (values cut at 2^-58 to 2^-60 of the largest, rounded products) is under half of that for these
    stencils.  The FP64 chain rounds at every tap and does not come near it."""
    st = stencil(name)
    dom = domain()
    arr = stencils.uniform(77, int(np.prod(dom.adims))).reshape(dom.adims)
    dom.set_field(0, arr)
    dom.upload()
    B.brickSweep(dom.brick(0), dom.brick(1), dom.dev_interior, st)
    B.synchronize()
    assert B.error_flags() == 0
    dom.download()
    got = dom.interior_view(dom.get_field(1))
    exact, chain = np.zeros(dom.n, np.longdouble), np.zeros(dom.n)
    for tap, c in zip(st.taps, st.coeff):
        v = arr[tuple(slice(dom.org[a] + tap[a], dom.org[a] + tap[a] + dom.n[a]) for a in range(3))]
        exact += np.longdouble(c) * v.astype(np.longdouble)
        chain += c * v
    once = np.sqrt(np.mean(np.spacing(np.abs(exact).astype(np.float64)) ** 2 / 12))
    rms = lambda x: float(np.sqrt(np.mean((x - exact).astype(np.float64) ** 2)))  # noqa: E731
    assert rms(chain) > 1.25 * once
    assert rms(got) < 1.25 * once, (rms(got) / once, rms(chain) / once)


@pytest.mark.parametrize("kind", ["zeros", "infinities", "wide"])
@pytest.mark.parametrize("name", ["star7", "star25", "star13-uneven"])
def test_star_kernels_agree_on_values_that_take_other_branches(name, kind, monkeypatch):
    st = stencil(name)
    dom = domain()
    arr = wide(dom.adims) if kind == "wide" else stencils.uniform(7, int(np.prod(dom.adims))).reshape(dom.adims)
    o = dom.org
    if kind == "zeros":
        arr[o[0] - 4:o[0] + 16] = 0.0
        arr[o[0]:o[0] + 4, o[1] + 3:o[1] + 20, o[2] + 5:o[2] + 30] = -0.0
        arr[o[0] + 9, o[1] + 10, o[2] + 11] = 1e-310
    elif kind == "infinities":
        arr[o[0] + 9, o[1] + 3, o[2] + 4] = np.inf
        arr[o[0] + 20, o[1] + 7, o[2] + 8] = -np.inf
    else:
        arr[:, :, :o[2] + 13] = stencils.uniform(9, arr[:, :, :o[2] + 13].size).reshape(arr[:, :, :o[2] + 13].shape)
    dom.set_field(0, arr)
    dom.upload()
    got = [_sweep_with(env, monkeypatch, dom, st, BK_ACC_NATIVE, dom.dev_interior) for env in KERNELS]
    for other in got[1:]:
        np.testing.assert_array_equal(got[0].view(np.uint8), other.view(np.uint8))
