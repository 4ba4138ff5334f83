"""The sign of zero sums on FP64 fields of zeros: -0 where every product is -0, else +0, as FP64
multiply-adds give it, also where bricks of zeros are not summed."""
import numpy as np
import pytest

from bricklib_gb300 import bricks as B, stencils
from bricklib_gb300._abi import BK_F64
from bricklib_gb300.domain import GridDomain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("signs", ["all positive", "all negative", "mixed"])
@pytest.mark.parametrize("zero", [0.0, -0.0])
@pytest.mark.parametrize("name", ["star7", "heat7", "star13", "star25", "cube27", "cube125"])
def test_sums_of_zeros_have_the_sign_of_fp64(name, zero, signs):
    st = stencils.make(name, 5)
    st.coeff = np.abs(st.coeff) * (-1.0 if signs == "all negative" else 1.0)
    if signs == "mixed":
        st.coeff = np.where(np.array([sum(map(abs, t)) for t in st.taps]) > 0, st.coeff, -st.coeff)
    dom = GridDomain((16, 24, 32), dtype=BK_F64)
    dom.set_field(0, np.full(dom.adims, zero))
    dom.upload()
    B.brickSweep(dom.brick(0), dom.brick(1), dom.dev_interior, st)
    B.synchronize()
    dom.download()
    got = dom.interior_view(dom.get_field(1))
    assert not got.any()
    assert (np.signbit(got) == all(np.signbit(c * zero) for c in st.coeff)).all()
