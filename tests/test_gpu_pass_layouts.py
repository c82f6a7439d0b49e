"""Forms that the two-sweep passes accept beside the plain ones: rows with padding (sj > ni, so that the last
lane of a row is a partial one), FP32 with lateral diffusion and with vertical sub-iterations, macro steps of
every scheme with tracer diffusion, and captured graphs. Each against its plain or one-sweep counterpart, bit
for bit: the same operations per face and cell, so the tolerance is 0."""
import numpy as np
import pytest

from code_b200 import cases
from code_b200 import getm as G
from code_b200 import state as S
from code_b200.getm import BcDevice, Context
from code_b200.grid import Grid, GetmDomain
from helpers import dev, host, make_ctx

pytestmark = pytest.mark.gpu

ARGS = ("uu", "vv", "ww", "hun", "hvn", "ho", "hn")
SCHEMES = [G.UPSTREAM, G.P2, G.SUPERBEE, G.MUSCL, G.P2_PDM]


class PaddedGrid(Grid):
    """The grid with `pad` unused elements at the end of every row."""

    def __init__(self, g, pad):
        super().__init__(g.nx, g.ny, g.kmax, g.dx, g.dy, g.imin, g.jmin)
        self.pad = pad

    def domain(self):
        sj = self.ni + self.pad
        return GetmDomain(self.imin, self.imax, self.jmin, self.jmax, self.kmax, sj, sj * self.nj, self.dx, self.dy,
                          self.ard1)


def _padded(a, pad, fill=np.nan):
    out = np.full(a.shape[:-1] + (a.shape[-1] + pad,), fill if a.dtype.kind == "f" else 0, a.dtype)
    out[..., :a.shape[-1]] = a
    return out


def _one_sweep(run):
    prev = G.set_vector_sweeps(False)
    try:
        return run()
    finally:
        G.set_vector_sweeps(prev)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("pad", [1, 2, 3, 4])
@pytest.mark.parametrize("nx", [53, 116, 121])
def test_padded_rows(nx, pad, dtype):
    c = cases.random_case(nx=nx, ny=33, kmax=5, seed=nx, dtype=dtype)

    def run(ctx, put):
        f, h, adv = dev(put(c["f"])), dev(put(np.zeros_like(c["f"]))), dev(put(np.zeros_like(c["f"])))
        ctx.do_advection_3d(c.par["dt"], f, *[dev(put(c[n])) for n in ARGS], G.HALFSPLIT, G.P2_PDM, G.P2_PDM, 2.0, G.H_TAG,
                            h, adv)
        return [host(x)[..., :c.grid.ni] for x in (f, h, adv)]

    wide = Context(PaddedGrid(c.grid, pad))
    wide.init_advection(*[dev(_padded(m, pad)) for m in c.masks()])
    for a, b in zip(run(wide, lambda x: _padded(x, pad)), run(make_ctx(c)[0], lambda x: x)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("pad", [1, 2])
def test_padded_rows_macro_step(pad, dtype):
    import torch

    c = S.baroclinic_case(nx=118, ny=33, kmax=6, recipe="islands", land=0.2, M=2, dt3=20.0, seed=5, dtype3=dtype)
    plain = BcDevice(c)
    t = {n: torch.from_numpy(_padded(host(a), pad, 0.0)).cuda() for n, a in plain.t.items()}
    st = BcDevice(tensors=t, pd=dict(c.pd), pi=dict(c.pi))
    wide = Context(PaddedGrid(c.grid, pad))
    wide.init_advection(*st.masks())
    wide.time_loop(st, 1, 4)
    make_ctx(c)[0].time_loop(plain, 1, 4)
    for n, a in plain.t.items():
        assert np.array_equal(host(st.t[n])[..., :c.grid.ni], host(a), equal_nan=True), n


@pytest.mark.parametrize("iters", [1, 3])
@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("size", [(53, 29), (116, 12), (118, 33)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_fp32_diffusion_and_sub_iterations(size, scheme, iters):
    c = cases.random_case(nx=size[0], ny=size[1], kmax=5, seed=size[1], dtype=np.float32)
    ctx, _ = make_ctx(c)
    arrs = [dev(c[n]) for n in ARGS]

    def run():
        f, h, adv = dev(c["f"]), dev(np.zeros_like(c["f"])), dev(np.zeros_like(c["f"]))
        ctx.do_advection_3d(c.par["dt"], f, *arrs, G.HALFSPLIT, scheme, scheme, 0.0 if iters > 1 else 3.0, G.H_TAG, h, adv,
                            iters)
        return [host(x) for x in (f, h, adv)]

    for a, b in zip(run(), _one_sweep(run)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("nx", [53, 116])
def test_macro_step_schemes(nx, scheme, dtype):
    c = S.baroclinic_case(nx=nx, ny=29, kmax=6, recipe="islands", land=0.2, M=2, dt3=20.0, seed=5, dtype3=dtype)
    for n in ("vel3d_adv_hor", "vel3d_adv_ver", "temp_adv_hor", "temp_adv_ver", "salt_adv_hor", "salt_adv_ver"):
        c.pi[n] = scheme
    c.pd["temp_AH"] = c.pd["salt_AH"] = 5.0
    rng = np.random.default_rng(1)
    c.f3["uu"][1:] += (0.3 * rng.normal(size=c.f3["uu"][1:].shape) * (c.au > 0)).astype(dtype)
    c.f3["vv"][1:] += (0.3 * rng.normal(size=c.f3["vv"][1:].shape) * (c.av > 0)).astype(dtype)
    ctx, _ = make_ctx(c)

    def run():
        st = BcDevice(c)
        ctx.time_loop(st, 1, 4)
        return {n: host(t) for n, t in st.t.items()}

    a, b = run(), _one_sweep(run)
    for n in a:
        assert np.array_equal(a[n], b[n], equal_nan=True), n


@pytest.mark.parametrize("kept", ["Tlo", "Slo"])
@pytest.mark.parametrize("nx", [53, 116])
def test_pair_with_one_carried_error_array(nx, kept):
    """The tracer pair with compensated storage of one tracer only, which keeps the one-sweep kernels."""
    c = S.baroclinic_case(nx=nx, ny=29, kmax=6, recipe="islands", land=0.2, M=2, dt3=20.0, seed=5, dtype3=np.float32)
    ctx, _ = make_ctx(c)

    def run():
        t = dict(BcDevice(c).t)
        del t["f3_Slo" if kept == "Tlo" else "f3_Tlo"]
        st = BcDevice(tensors=t, pd=dict(c.pd), pi=dict(c.pi))
        ctx.time_loop(st, 1, 4)
        return {n: host(a) for n, a in t.items()}

    a, b = run(), _one_sweep(run)
    for n in a:
        assert np.array_equal(a[n], b[n], equal_nan=True), n


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_captured_steps(dtype):
    """A captured time loop and tracer step (chained launches become edges of the graph) replayed."""
    import torch

    c = S.baroclinic_case(nx=53, ny=29, kmax=6, recipe="islands", land=0.2, M=2, dt3=20.0, seed=5, dtype3=dtype)
    ctx, _ = make_ctx(c)
    st = BcDevice(c)
    start = {n: t.clone() for n, t in st.t.items()}
    tracer = [st.t["f3_" + n].clone() for n in ("T", "uu", "vv", "ww", "hun", "hvn", "ho", "hn", "nuh")]

    def steps():
        ctx.time_loop(st, 1, 4)
        ctx.tracer_step(20.0, *tracer, G.HALFSPLIT, G.P2_PDM, G.P2_PDM, 0.0, 0.9, 1e-9)

    ipar = list(st.c.ipar)
    steps()
    want = [host(t) for t in (*st.t.values(), *tracer)]
    first = tracer[0].clone()
    torch.cuda.synchronize()
    for n, t in start.items():
        st.t[n].copy_(t)
    tracer[0].copy_(start["f3_T"])
    st.c.ipar[:] = ipar
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.set_stream(torch.cuda.current_stream())
        steps()
    graph.replay()
    torch.cuda.synchronize()
    assert not torch.equal(first, start["f3_T"])
    for a, b in zip((*st.t.values(), *tracer), want):
        assert np.array_equal(host(a), b, equal_nan=True)
