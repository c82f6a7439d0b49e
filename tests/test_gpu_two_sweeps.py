"""The two-sweep passes of a HALFSPLIT advection (adv_fused.cuh) at the edges of their strips and row
segments, against the oracle (FP64) and against the one-sweep kernels (FP32), bit for bit.

Both evaluate every face flux and cell update with the same operations, so the tolerance is 0. A strip
owns 28 columns (one cell per lane), 60 or 58 (two) or 120 (four); a row segment 8 to 64 rows, four
segments per block. Rows of 4n, 4n+2 and odd length take four, two and one cell per lane in FP32.
"""
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
# (nx, ny): rows of nx + 4 cells
SIZES = [(1, 1), (24, 3), (25, 4), (52, 36), (53, 29), (112, 5), (116, 61), (117, 7), (118, 33), (121, 28)]


@pytest.mark.parametrize("scheme", [G.UPSTREAM, G.P2, G.SUPERBEE, G.MUSCL, G.P2_PDM])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("tag", [G.H_TAG, G.U_TAG, G.V_TAG, G.W_TAG])
def test_halfsplit_fp64_equals_oracle(size, scheme, tag):
    c = cases.random_case(nx=size[0], ny=size[1], kmax=5, seed=size[0] + tag)
    ctx, _ = make_ctx(c)
    f, hires, adv = c["f"].copy(), np.zeros_like(c["f"]), np.zeros_like(c["f"])
    AH = 2.0 if scheme == G.MUSCL else 0.0
    tf, th, ta = dev(f), dev(hires), dev(adv)
    oracle.Oracle(c.grid).do_advection_3d(c.masks(), c.par["dt"], f, *[c[n] for n in ARGS], G.HALFSPLIT, scheme, scheme,
                                          AH, tag, hires, adv)
    ctx.do_advection_3d(c.par["dt"], tf, *[dev(c[n]) for n in ARGS], G.HALFSPLIT, scheme, scheme, AH, tag, th, ta)
    assert np.array_equal(host(tf), f)
    assert np.array_equal(host(th), hires)
    assert np.array_equal(host(ta), adv)


def _both(run):
    """run() with the two-sweep passes and with the one-sweep kernels."""
    a = run()
    G.set_vector_sweeps(False)
    try:
        b = run()
    finally:
        G.set_vector_sweeps(True)
    return a, b


@pytest.mark.parametrize("scheme", [G.UPSTREAM, G.P2, G.SUPERBEE, G.MUSCL, G.P2_PDM])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_halfsplit_fp32_equals_one_sweep_kernels(size, scheme):
    c = cases.random_case(nx=size[0], ny=size[1], kmax=5, seed=size[1], dtype=np.float32)
    ctx, _ = make_ctx(c)
    arrs = [dev(c[n]) for n in ARGS]

    def run():
        f, h, adv = dev(c["f"]), dev(np.zeros_like(c["f"])), dev(np.zeros_like(c["f"]))
        ctx.do_advection_3d(c.par["dt"], f, *arrs, G.HALFSPLIT, scheme, scheme, 0.0, G.H_TAG, h, adv)
        return [host(x) for x in (f, h, adv)]

    for a, b in zip(*_both(run)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("size", [(20, 9), (53, 29), (116, 12), (118, 33), (121, 70)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_macro_step_equals_one_sweep_kernels(size, dtype):
    """Momentum advection formed from uu, vv, ww, the tracer pair and its carried errors."""
    c = S.baroclinic_case(nx=size[0], ny=size[1], kmax=6, recipe="islands", land=0.2, M=2, dt3=20.0, seed=5, dtype3=dtype)
    rng = np.random.default_rng(1)
    c.f3["uu"][1:] += (0.3 * rng.normal(size=c.f3["uu"][1:].shape) * (c.au > 0)).astype(dtype)
    c.f3["vv"][1:] += (0.3 * rng.normal(size=c.f3["vv"][1:].shape) * (c.av > 0)).astype(dtype)
    ctx, _ = make_ctx(c)

    def run():
        st = BcDevice(c)
        ctx.time_loop(st, 1, 4)
        return {n: host(t) for n, t in st.t.items()}

    a, b = _both(run)
    for n in a:
        assert np.array_equal(a[n], b[n], equal_nan=True), n
