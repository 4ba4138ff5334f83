"""The 27-point cube without mirror symmetry on FP32 / BF16 storage, streamed along runs of i-adjacent
list entries: a brick's last column waits for the brick after it where the run goes on.  Every brick
has the same bits whatever runs the list makes of it, and meets the storage type's bound against the
oracle; output bricks off the vector boundary take element stores.

Bounds: 27 products, at most 11 additions in a row: n 2^-24 of the largest sum of terms is below 1e-5;
BF16 adds its output's rounding, 2^-8."""
import numpy as np
import pytest

from bricklib_gb300 import bricks as B, stencils
from bricklib_gb300._abi import BK_BF16, BK_F32
from bricklib_gb300.domain import GridDomain
from oracle import oracle

pytestmark = pytest.mark.gpu


def lists(dom, rng):
    it = np.asarray(dom.interior, dtype=np.uint32)
    cuts = np.cumsum(rng.integers(1, 6, size=len(it)))
    pieces = np.split(it, cuts[cuts < len(it)])
    return {"grid": it, "shuffled": rng.permutation(it), "one": it[-1:], "two": it[:2],
            "pieces": np.concatenate([pieces[p] for p in rng.permutation(len(pieces))]),
            "repeats": np.repeat(it[:50], rng.integers(1, 3, size=min(50, len(it)))), "tail": it[3:3 + 61]}


@pytest.mark.parametrize("off", [0, 2])
@pytest.mark.parametrize("dtype", [BK_F32, BK_BF16])
@pytest.mark.parametrize("n", [(16, 16, 8), (24, 40, 72), (32, 64, 256)])  # (k, j, i): runs of 1, 9 and 32 bricks
def test_cube27_stream_same_bits_for_every_list(n, dtype, off):
    st = stencils.make("cube27", 3)
    dom = GridDomain(n, dtype=dtype)
    arr = stencils.uniform(19, int(np.prod(dom.adims))).reshape(dom.adims)
    dom.set_field(0, arr)
    dom.upload()
    x = arr.astype(np.float32).astype(np.float64) if dtype == BK_F32 else \
        B.bf16_to_f32(B.f32_to_bf16(arr.astype(np.float32))).astype(np.float64)
    want, o = np.zeros_like(x), dom.org
    oracle.array_sweep(x, want, tuple(o), tuple(a + b for a, b in zip(o, n)), st.offsets(), st.coeff)
    step, size = 2 * dom.bsize, dom.bsize
    host = np.empty(dom.nbricks * step, dom.storage.host.dtype)
    full = None
    for key, lst in lists(dom, np.random.default_rng(2)).items():
        host.view(np.uint8)[:] = 0xFF
        out = B.movBrickStorage(B.BrickStorage(dom.nbricks, step, dtype, host=host.copy()), to_device=True)
        B.brickSweep(dom.brick(0), B.Brick(dom.brick(0).bInfo, out, off), B.BrickList(np.ascontiguousarray(lst)), st)
        B.synchronize()
        assert B.error_flags() == 0
        back = B.movBrickStorage(out, to_device=False).host.reshape(dom.nbricks, step)
        got, rest = back[:, off:off + size], np.delete(back, np.s_[off:off + size], axis=1)
        assert np.all(rest.view(np.uint8) == 0xFF)
        listed = np.unique(lst)
        assert int((got.view(np.uint8) != 0xFF).any(axis=1).sum()) == len(listed)
        if full is None:
            full = got.copy()
            dom.storage.host.reshape(dom.nbricks, dom.nfields, -1)[:, 1, :] = full
            a, b = dom.interior_view(dom.get_field(1)), dom.interior_view(want)
            assert np.linalg.norm(a - b) <= (1e-5 if dtype == BK_F32 else 2.0 ** -7) * np.linalg.norm(b)
        np.testing.assert_array_equal(got[listed].view(np.uint8), full[listed].view(np.uint8), err_msg=key)
