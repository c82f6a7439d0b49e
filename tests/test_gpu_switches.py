"""The process-wide choice of the sweep kernels turned by another thread while a step runs: both choices
give the same values, so neither the step's result nor its success may depend on when it is turned."""
import threading

import numpy as np
import pytest

from code_b200 import getm as G
from code_b200 import state as S
from code_b200.getm import BcDevice
from helpers import host, make_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_switch_turned_during_macro_steps(dtype):
    c = S.baroclinic_case(nx=20, ny=9, kmax=6, recipe="islands", land=0.2, M=1, dt3=5.0, seed=5, dtype3=dtype)
    ctx, _ = make_ctx(c)
    st = BcDevice(c)
    ctx.time_loop(st, 1, 300)
    want = {n: host(t) for n, t in st.t.items()}
    stop = threading.Event()

    def turn():
        on = False
        while not stop.is_set():
            G.set_vector_sweeps(on)
            on = not on

    t = threading.Thread(target=turn)
    t.start()
    try:
        st = BcDevice(c)
        ctx.time_loop(st, 1, 300)
    finally:
        stop.set()
        t.join()
        G.set_vector_sweeps(True)
    for n in want:
        assert np.array_equal(host(st.t[n]), want[n], equal_nan=True), n
