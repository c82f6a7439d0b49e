"""The micro-step loop's fused launches (both momentum-advection components with the bottom friction,
Coriolis terms inside the velocity updates, sealevel + depth_update) against the separate launches,
bit for bit: the same expressions per point, so the tolerance is 0. Sizes at the edges of the small
(24 x 8) and the large (56 x 16) tiles of the momentum advection, closed and with open boundaries on
every side, with and without the barotropic roughness."""
import numpy as np
import pytest

from code_b200 import getm as G
from code_b200 import state as S
from code_b200.getm import BcDevice
from helpers import host, make_ctx

pytestmark = pytest.mark.gpu


def _sides(nx, ny):
    return S.OpenBoundaries(west=[(1, 2, ny - 1, S.CLAMPED)], north=[(ny, 3, nx - 3, S.SOMMERFELD)],
                            east=[(nx, 2, ny - 1, S.ZERO_GRADIENT)], south=[(1, 4, nx - 2, S.CLAMPED)], ramp=10, amp=0.2,
                            phase=0.4, period=4000.0)


@pytest.mark.parametrize("runtype", [1, 4])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("bdy", [False, True], ids=["closed", "open"])
@pytest.mark.parametrize("size", [(20, 4), (21, 13), (44, 12), (45, 28), (690, 196)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_fused_micro_steps_equal_separate_launches(size, bdy, dtype, runtype):
    nx, ny = size
    b = _sides(nx, ny) if bdy and ny > 8 else None
    c = S.baroclinic_case(nx=nx, ny=ny, kmax=2, recipe="shelf", M=3, dt3=9.0, seed=7, dtype3=dtype, bdy=b)
    c.pi["runtype"] = runtype
    rng = np.random.default_rng(2)
    c.f2["U"] += 0.5 * rng.normal(size=c.f2["U"].shape) * (c.au > 0)
    c.f2["V"] += 0.5 * rng.normal(size=c.f2["V"].shape) * (c.av > 0)
    ctx, _ = make_ctx(c)
    if b is not None:
        ctx.set_open_boundaries(b)
    out = []
    prev = G.set_fused_micro_step(True)
    try:
        for on in (True, False):
            G.set_fused_micro_step(on)
            st = BcDevice(c)
            ctx.time_loop(st, 1, 7)
            out.append({n: host(t) for n, t in st.t.items()})
    finally:
        G.set_fused_micro_step(prev)
    for n in out[0]:
        assert np.array_equal(out[0][n], out[1][n], equal_nan=True), n
