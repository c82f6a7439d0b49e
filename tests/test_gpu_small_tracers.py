"""FP32 advection of a tracer in the subnormal range: the field times 2^-127 advances as the field itself
does, to the spacing of the subnormal numbers.

UPSTREAM and P2 are linear, so scaling by a power of two changes nothing but the roundings: the field is
at most 1.01, so every scaled value is subnormal and sums of them are exact; products and quotients are
off by half of u = 2^-149, their spacing. With |U| <= 1, CFL <= 0.02, h = 1 and dt = 10: the face value is
off by u, the flux by 1.5 u, the flux divergence (over 500 m) by 0.51 u, dt times it by 5.6 u, the increment by
6.6 u; as much again for the (finer) roundings of the unscaled run, 14 u per sweep; five sweeps that amplify
by at most 1.1 each stay below 128 u. Divisions that flush subnormal numbers would leave the field as it
was: off by its movement, about 6e-4 or 2500 u.
"""
import numpy as np
import pytest

from code_b200 import cases
from code_b200 import getm as G
from helpers import dev, host, make_ctx

pytestmark = pytest.mark.gpu

ARGS = ("uu", "vv", "ww", "hun", "hvn", "ho", "hn")


@pytest.mark.parametrize("vector", [True, False], ids=["passes", "tiles"])
@pytest.mark.parametrize("scheme", [G.UPSTREAM, G.P2])
@pytest.mark.parametrize("nx", [50, 52, 53])
def test_subnormal_increments_are_kept(nx, scheme, vector):
    c = cases.tracer_rotation(nx=nx, ny=44, kmax=5, depth=5.0, dt=10.0, dtype=np.float32)
    rng = np.random.default_rng(nx)
    c["ww"][1:-1] = (1e-4 * rng.normal(size=c["ww"][1:-1].shape) * (c["az"] == 1)).astype(np.float32)
    ctx, _ = make_ctx(c)
    arrs = [dev(c[n]) for n in ARGS]
    small = (c["f"] * np.float32(2.0 ** -127)).astype(np.float32)
    out = []
    prev = G.set_vector_sweeps(vector)
    try:
        for f0 in (small, (small.astype(np.float64) * 2.0 ** 127).astype(np.float32)):
            f = dev(f0)
            ctx.do_advection_3d(c.par["dt"], f, *arrs, G.HALFSPLIT, scheme, scheme, 0.0, G.H_TAG)
            out.append(host(f).astype(np.float64))
    finally:
        G.set_vector_sweeps(prev)
    assert np.abs(out[1] - c["f"]).max() > 1e-4  # the field moves
    err = np.abs(out[0] * 2.0 ** 127 - out[1]).max() * 2.0 ** (149 - 127)
    assert err <= 128, err
