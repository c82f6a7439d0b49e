"""The two-sweep passes on few rows and on every remainder of the levels over the warps of a block (two
levels), one to nine levels: FP64 against the oracle, FP32 against the one-sweep kernels, bit for bit (the
same operations per face and cell, so the tolerance is 0)."""
import numpy as np
import pytest

import oracle
from code_b200 import cases
from code_b200 import getm as G
from code_b200 import state as S
from code_b200.getm import BcDevice
from helpers import dev, host, make_ctx

pytestmark = pytest.mark.gpu

ARGS = ("uu", "vv", "ww", "hun", "hvn", "ho", "hn")


@pytest.mark.parametrize("kmax", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("size", [(30, 1), (57, 2), (116, 9), (121, 30)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_levels_fp64_equals_oracle(size, kmax):
    c = cases.random_case(nx=size[0], ny=size[1], kmax=kmax, seed=kmax)
    ctx, _ = make_ctx(c)
    f, hires, adv = c["f"].copy(), np.zeros_like(c["f"]), np.zeros_like(c["f"])
    tf, th, ta = dev(f), dev(hires), dev(adv)
    oracle.Oracle(c.grid).do_advection_3d(c.masks(), c.par["dt"], f, *[c[n] for n in ARGS], G.HALFSPLIT, G.P2_PDM, G.P2_PDM,
                                          0.0, G.H_TAG, hires, adv)
    ctx.do_advection_3d(c.par["dt"], tf, *[dev(c[n]) for n in ARGS], G.HALFSPLIT, G.P2_PDM, G.P2_PDM, 0.0, G.H_TAG, th, ta)
    assert np.array_equal(host(tf), f)
    assert np.array_equal(host(th), hires)
    assert np.array_equal(host(ta), adv)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kmax", [2, 3, 5])
@pytest.mark.parametrize("size", [(250, 1), (118, 9)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_levels_macro_step_equals_one_sweep_kernels(size, kmax, dtype):
    c = S.baroclinic_case(nx=size[0], ny=size[1], kmax=kmax, recipe="islands", land=0.2, M=2, dt3=20.0, seed=5, dtype3=dtype)
    ctx, _ = make_ctx(c)
    out = []
    try:
        for on in (True, False):
            G.set_vector_sweeps(on)
            st = BcDevice(c)
            ctx.time_loop(st, 1, 4)
            out.append({n: host(t) for n, t in st.t.items()})
    finally:
        G.set_vector_sweeps(True)
    for n in out[0]:
        assert np.array_equal(out[0][n], out[1][n], equal_nan=True), n
