"""Column kernels whose dynamic shared memory depends on kmax: the largest kmax admitted, the first one
refused, and contexts of different kmax launching from different host threads at the same time (the
opt-in limit belongs to the kernel, not to the context)."""
import threading

import numpy as np
import pytest

import oracle
from code_b200 import state as S
from code_b200.getm import BcDevice, Context, GetmError
from code_b200.grid import Grid
from helpers import dev, host, make_ctx

pytestmark = pytest.mark.gpu


def _system(kmax, ncol, seed):
    rng = np.random.default_rng(seed)
    au, cu = -rng.random((kmax + 1, ncol)), -rng.random((kmax + 1, ncol))
    return au, 1.5 - au - cu, cu, rng.normal(size=(kmax + 1, ncol))


def test_tridiagonal_largest_kmax():
    kmax, ncol = 199, 33
    sys_ = _system(kmax, ncol, 1)
    g = Grid(4, 4, kmax, 1.0, 1.0)
    value = dev(np.zeros((kmax + 1, ncol)))
    Context(g).tridiagonal(kmax, 0, kmax, *[dev(a) for a in sys_], value)
    o = oracle.Oracle(g)
    for q in range(ncol):
        assert np.array_equal(host(value)[:, q], o.tridiagonal(kmax, 0, kmax, *[np.ascontiguousarray(a[:, q]) for a in sys_]))
    big = [dev(a) for a in _system(kmax + 1, ncol, 1)]
    with pytest.raises(GetmError, match="kmax too large"):
        Context(g).tridiagonal(kmax + 1, 0, kmax + 1, *big, dev(np.zeros((kmax + 2, ncol))))


def _threads(jobs, calls):
    """Each job (its own context and stream) called `calls` times on a thread of its own; the errors."""
    errors, start = [], threading.Barrier(len(jobs))

    def loop(job):
        start.wait()
        for _ in range(calls):
            try:
                job()
            except GetmError as e:
                errors.append(str(e))
                return

    threads = [threading.Thread(target=loop, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def test_tridiagonal_threads_of_different_kmax():
    import torch

    jobs, keep = [], []
    for kmax in (100, 199, 110, 190):
        stream = torch.cuda.Stream()
        ctx = Context(Grid(4, 4, kmax, 1.0, 1.0), stream)
        arrs = [dev(a) for a in _system(kmax, 1, kmax)] + [dev(np.zeros((kmax + 1, 1)))]
        keep.append((stream, ctx, arrs))
        jobs.append(lambda ctx=ctx, kmax=kmax, arrs=arrs: ctx.tridiagonal(kmax, 0, kmax, *arrs))
    torch.cuda.synchronize()
    errors = _threads(jobs, 30000)
    torch.cuda.synchronize()
    assert not errors, errors


@pytest.mark.parametrize("dtype,kmaxs", [(np.float64, (150, 199)), (np.float32, (5, 63))], ids=["fp64", "fp32"])
def test_macro_steps_on_threads_of_different_kmax(dtype, kmaxs):
    """Pressure integral (FP64 above 48 KB from kmax 149 on) and 3D momentum solve (FP32, kmax < 64)."""
    import torch

    jobs, keep = [], []
    for kmax in kmaxs * 2:
        c = S.baroclinic_case(nx=8, ny=6, kmax=kmax, recipe="shelf", M=1, dt3=1.0, seed=kmax, dtype3=dtype)
        ctx, _ = make_ctx(c)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        ctx.set_stream(stream)
        st = BcDevice(c)
        keep.append((stream, ctx, st))
        n = [0]

        def step(ctx=ctx, st=st, n=n):
            n[0] += 1
            if dtype is np.float64:
                ctx.internal_pressure(st)
            else:
                ctx.time_loop(st, n[0], 1)

        jobs.append(step)
    torch.cuda.synchronize()
    errors = _threads(jobs, 8000 if dtype is np.float64 else 400)
    torch.cuda.synchronize()
    assert not errors, errors
