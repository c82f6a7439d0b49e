"""The size rule of the two-sweep passes (two_sweeps_pay) for a tracer step and a recorded one: which form
runs on either side of its lines (2^20, 2^21 and 2^23 elements) for odd and even rows, FP64 and FP32, with and
without diffusion -- and that the field (and tape) are those of the one-sweep kernels, bit for bit (the same
operations per face and cell, so the tolerance is 0)."""
import numpy as np
import pytest

from code_b200 import cases
from code_b200 import getm as G
from code_b200.getm import Context
from code_b200.grid import Grid
from helpers import dev

pytestmark = pytest.mark.gpu

ARGS = ("uu", "vv", "ww", "hun", "hvn", "ho", "hn", "nuh")
SIZES = {"small": (300, 200, 3), "small_odd": (301, 199, 3), "middle": (600, 520, 3), "middle_odd": (601, 519, 3),
         "between": (1000, 700, 3), "between_odd": (1001, 699, 3), "large": (1700, 1300, 3), "large_odd": (1701, 1299, 3)}


def _expected(size, f64, AH, rec):
    between, odd = size.startswith("between"), size.endswith("odd")
    if f64:
        return size == "small" if AH > 0 and not odd else not between
    return rec or odd or (AH == 0 and not between)


def _problem(size, dtype):
    import torch

    nx, ny, kmax = SIZES[size]
    g = Grid(nx, ny, kmax, 500.0, 500.0)
    rng = np.random.default_rng(nx)
    az = np.zeros(g.shape2(), np.int32)
    az[g.interior()] = rng.random((ny, nx)) > 0.2
    au, av, ax = cases.derive_uvx(az)
    ctx = Context(g)
    ctx.init_advection(*[dev(m) for m in (az, au, av, ax)])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(ny)
    rnd = lambda: torch.randn(g.shape3(), generator=gen, device="cuda", dtype=dtype)  # noqa: E731
    t = {n: 1.0 + 0.2 * torch.sin(rnd()) for n in ("hun", "hvn", "ho")}
    t.update(uu=0.5 * rnd(), vv=0.5 * rnd(), ww=1e-4 * rnd(), hn=t["ho"].clone(), nuh=1e-3 * torch.abs(rnd()))
    return ctx, [t[n] for n in ARGS], 10.0 + rnd()


@pytest.mark.parametrize("AH", [0.0, 20.0])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("size", SIZES)
def test_route_and_result(size, prec, AH):
    import torch

    dtype = torch.float64 if prec == "fp64" else torch.float32
    ctx, args, f0 = _problem(size, dtype)
    tail = (G.HALFSPLIT, G.P2_PDM, G.P2_PDM, AH, 0.9, 1e-9)
    ctx.timers(enable=True, reset=True)
    f = f0.clone()
    ctx.tracer_step(30.0, f, *args, *tail)
    assert ("adv_split_uv" in ctx.timers(reset=True)) == _expected(size, prec == "fp64", AH, False)
    tape = ctx.tape(dtype)
    tape[0].zero_()
    fr = f0.clone()
    ctx.tracer_step_record(30.0, fr, *args, *tail, tape)
    launches = ctx.timers(reset=True)["tracer_record"][1]  # sweeps, tape copy, diffusion
    assert launches == (5 if _expected(size, prec == "fp64", AH, True) else 7)
    prev = G.set_vector_sweeps(False)
    try:
        one, rec = f0.clone(), f0.clone()
        ctx.tracer_step(30.0, one, *args, *tail)
        tape1 = ctx.tape(dtype)
        tape1[0].zero_()
        ctx.tracer_step_record(30.0, rec, *args, *tail, tape1)
    finally:
        G.set_vector_sweeps(prev)
    assert not torch.equal(f, f0)
    for a, b in ((f, one), (fr, rec), (fr, f), (tape[0], tape1[0]), (tape[1], tape1[1])):
        assert torch.equal(a, b)
