"""Blumberg-Mellor internal pressure at the edges of its level groups (4) and blocks (32 x 4): FP64, the
oracle's expressions in its order, so the tolerance is 0."""
import numpy as np
import pytest

import oracle
from code_b200 import state as S
from code_b200.getm import BcDevice
from helpers import host, make_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kmax", [1, 2, 3, 4, 5, 6, 8, 9, 13])
@pytest.mark.parametrize("size", [(28, 4), (29, 5), (61, 27)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_blumberg_mellor_groups(kmax, size):
    c = S.baroclinic_case(nx=size[0], ny=size[1], kmax=kmax, recipe="islands", land=0.2, M=2, dt3=20.0, seed=kmax)
    c.f3["idpdx"][...] = 3.0
    c.f3["idpdy"][...] = 4.0
    ctx, _ = make_ctx(c)
    st = BcDevice(c)
    ctx.internal_pressure(st)
    oracle.bc_call(c, "internal_pressure")
    for n in ("idpdx", "idpdy"):
        assert np.array_equal(host(st.t["f3_" + n]), c.f3[n]), n
