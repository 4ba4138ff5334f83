"""The 27-point cube without mirror symmetry on FP32 / BF16 storage takes two kernels, by the length
of the brick list: streamed along runs of bricks on long ones, column pairs on short ones.  A brick
has the same bits from both, whatever runs the list makes, on re-pointed adjacency and beside
entries that cannot run; so have the FP64 cubes whose class sums are streamed."""
import numpy as np
import pytest

from bricklib_gb300 import bricks as B, stencils
from bricklib_gb300._abi import BK_ACC_NATIVE, BK_BF16, BK_F32, BK_F64
from bricklib_gb300.domain import GridDomain
from oracle import oracle
from test_gpu_sweep import _istream_stencil, _sweep_with

pytestmark = pytest.mark.gpu

LONG = 20000  # entries: more than 2.5 per resident CTA (2128 of FP32, 2432 of BF16 storage)


def tiled(lst):
    return np.ascontiguousarray(np.tile(lst, -(-LONG // len(lst))).astype(np.uint32))


def bits(out, dom, ids):
    return np.ascontiguousarray(out.reshape(dom.nbricks, dom.nfields, -1)[ids, 1, :]).view(np.uint8)


def shuffled(it):
    """No two i-neighbours in a row: no run continues."""
    return np.concatenate([it[q::5] for q in range(5)])


@pytest.mark.parametrize("dtype", [BK_F32, BK_BF16])
def test_cube27_long_and_short_lists_same_bits(dtype, monkeypatch):
    st = stencils.make("cube27", 3)
    n = (64, 128, 512)  # 8192 bricks in runs of 64
    dom = GridDomain(n, dtype=dtype)
    arr = stencils.uniform(19, int(np.prod(dom.adims))).reshape(dom.adims)
    dom.set_field(0, arr)
    it = np.asarray(dom.interior, dtype=np.uint32)
    rng = np.random.default_rng(4)
    cuts = np.cumsum(rng.integers(1, 9, size=len(it)))
    pieces = np.split(it, cuts[cuts < len(it)])
    lists = {"grid": it, "shuffled": rng.permutation(it), "pieces": np.concatenate([pieces[p] for p in rng.permutation(len(pieces))]),
             "short": it[1000:3000], "one": it[-1:]}
    full = None
    for key, lst in lists.items():
        out = _sweep_with(None, monkeypatch, dom, st, BK_ACC_NATIVE, B.BrickList(np.ascontiguousarray(lst)))
        if full is None:
            full = out
            got = dom.interior_view(dom.get_field(1)).astype(np.float64)
        np.testing.assert_array_equal(bits(out, dom, lst), bits(full, dom, lst), err_msg=key)
        written = out.view(np.uint8).reshape(dom.nbricks, dom.nfields, -1)[:, 1, :]
        assert int((written != 0xFF).any(axis=1).sum()) == len(lst), key
    x = arr.astype(np.float32).astype(np.float64) if dtype == BK_F32 else \
        B.bf16_to_f32(B.f32_to_bf16(arr.astype(np.float32))).astype(np.float64)
    want, o = np.zeros_like(x), dom.org
    oracle.array_sweep(x, want, tuple(o), tuple(a + b for a, b in zip(o, n)), st.offsets(), st.coeff)
    want = dom.interior_view(want)
    # 27 products, at most 11 additions in a row; BF16 rounds its output too
    assert np.linalg.norm(got - want) <= (1e-5 if dtype == BK_F32 else 2.0 ** -7) * np.linalg.norm(want)


CUBES = [(BK_F32, "cube27"), (BK_BF16, "cube27"), (BK_F64, "sym27"), (BK_F64, "sym27kj"), (BK_F64, "sym125"),
         (BK_F64, "sym125ij"), (BK_F64, "cube125")]


def make(name):
    return stencils.make("cube27", 11) if name == "cube27" else _istream_stencil(name)


def repointed(dom, seed):
    """i-lo, diagonal and i-hi entries of some bricks re-pointed, and some bricks their own i neighbours."""
    adj = dom.bInfo.adj.copy()
    rng = np.random.default_rng(seed)
    it = dom.interior
    for slot, frac in ((12, 5), (3, 6), (23, 6), (11, 7), (14, 9)):
        v = rng.choice(it, size=len(it) // frac, replace=False)
        adj[v, slot] = rng.choice(it, size=len(v))
    own = rng.choice(it, size=len(it) // 7, replace=False)
    adj[own, 14] = own
    adj[own[::2], 12] = own[::2]
    return adj


@pytest.mark.parametrize("dtype,name", CUBES)
def test_streamed_cubes_follow_repointed_adjacency(dtype, name, monkeypatch):
    st = make(name)
    dom = GridDomain((32, 64, 64), device=False, dtype=dtype)
    dom.bInfo = B.BrickInfo(dom.nbricks, repointed(dom, 12))
    arr = stencils.uniform(8, int(np.prod(dom.adims))).reshape(dom.adims)
    dom.set_field(0, arr)
    dom.to_device()
    it = np.asarray(dom.interior, dtype=np.uint32)
    want = bits(_sweep_with(None, monkeypatch, dom, st, BK_ACC_NATIVE, B.BrickList(shuffled(it))), dom, it)
    for lst in (it, tiled(it), tiled(shuffled(it))):
        got = bits(_sweep_with(None, monkeypatch, dom, st, BK_ACC_NATIVE, B.BrickList(lst)), dom, it)
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("dtype,name", CUBES)
def test_streamed_cubes_beside_entries_that_cannot_run(dtype, name, monkeypatch):
    """List entries beyond the bricks, bricks whose own storage index is out of range and neighbours
    out of range, inside runs: the flag is raised, those bricks are not written, neighbours out of
    range read brick 0, and every other brick has the bits it has in a list without runs."""
    st = make(name)
    dom = GridDomain((32, 64, 64), device=False, dtype=dtype)
    adj = dom.bInfo.adj.copy()
    rng = np.random.default_rng(13)
    it = np.asarray(dom.interior, dtype=np.uint32)
    dead = rng.choice(it, size=len(it) // 9, replace=False)
    adj[dead, 13] = dom.nbricks + 5
    lost = rng.choice(it, size=len(it) // 6, replace=False)
    adj[lost, rng.choice([3, 5, 12, 14, 22], size=len(lost))] = 0xFFFFFFF0
    dom.bInfo = B.BrickInfo(dom.nbricks, adj)
    arr = stencils.uniform(9, int(np.prod(dom.adims))).reshape(dom.adims)
    dom.set_field(0, arr)
    dom.to_device()
    alive = np.setdiff1d(it, dead)

    def swept(lst):
        raw = dom.storage.host.view(np.uint8).reshape(dom.nbricks, dom.nfields, -1)
        raw[:, 1, :] = 0xFF
        dom.upload()
        B.error_flags()
        B.brickSweep(dom.brick(0), dom.brick(1), B.BrickList(np.ascontiguousarray(lst.astype(np.uint32))), st)
        B.synchronize()
        assert B.error_flags() == 1
        dom.download()
        out = dom.storage.host.copy()
        written = (out.view(np.uint8).reshape(dom.nbricks, dom.nfields, -1)[:, 1, :] != 0xFF).any(axis=1)
        assert np.array_equal(np.flatnonzero(written), np.sort(alive))
        return bits(out, dom, alive)

    with_bad = np.insert(it.astype(np.int64), rng.integers(0, len(it), 60), dom.nbricks + rng.integers(0, 1000, 60))
    want = swept(shuffled(it))
    for lst in (with_bad, tiled(with_bad), tiled(it)):
        np.testing.assert_array_equal(swept(lst), want)
