"""A call on a caller's stream comes after everything the caller queued there, also behind a
kernel that starts its dependents early without having waited itself (programmatic dependent
launch): the first kernel of a call is an ordinary launch on such a stream."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

from ppm_b200 import build as B
from ppm_b200 import capi
from ppm_b200 import harness as H
from parity_util import random_state

pytestmark = pytest.mark.gpu

SLOW = 4_000_000  # cycles, about 2 ms


@pytest.fixture(scope="module")
def queue(tmp_path_factory):
    so = tmp_path_factory.mktemp("caller") / "libcaller.so"
    subprocess.run([B.nvcc(), *B.ARCH, "-shared", "-Xcompiler", "-fPIC", "-o", str(so),
                    str(Path(__file__).with_name("caller_stream.cu"))], check=True)
    fn = C.CDLL(str(so)).queue_slow_copy
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_longlong, C.c_longlong, C.c_void_p]
    return fn


@pytest.mark.parametrize("call", ["solve", "level", "sweep", "boundary", "pressure", "timestep",
                                  "expansion"])
def test_call_waits_for_the_callers_work(queue, call):
    torch = pytest.importorskip("torch")
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    g = H.Grid.uniform((16, 14, 12))
    f = random_state(g, hp, seed=4)
    stream = torch.cuda.Stream()
    ctx = capi.Context(0, stream=stream.cuda_stream)
    outs = []
    for slow in (False, True):
        fd = {k: torch.from_numpy(v.copy()).cuda() for k, v in f.items()}
        d = fd["d"].clone()
        press = torch.ones(g.shape, dtype=torch.float64, device="cuda")
        dt = torch.zeros(1, dtype=torch.float64, device="cuda")
        if slow:
            fd["d"].fill_(1.0)  # until the slow kernel has written the densities
        torch.cuda.synchronize()
        if slow:
            assert queue(fd["d"].data_ptr(), d.data_ptr(), g.size, SLOW, stream.cuda_stream) == 0
        dev = dict(memory=capi.MEM_DEVICE)
        if call == "solve":
            ctx.solve_ppm_de(g, hp, 1e-3, 0, fd, want_stats=False, **dev)
        elif call == "level":
            ctx.solve_level([g], hp, 1e-3, 0, [fd])
        elif call == "sweep":
            ctx.euler_sweep(0, g, hp, 1e-3, fd, press, **dev)
        elif call == "boundary":
            ctx.set_boundary(g, fd, True)
        elif call == "pressure":
            ctx.compute_pressure(g, hp, fd, press, **dev)
        elif call == "timestep":
            ctx.compute_timestep(g, hp, fd, dt_device=dt, want_host=False, **dev)
        else:
            ctx.expansion_terms(g, hp, fd, None, 1.0, 1.0, 0.1, **dev)
        torch.cuda.synchronize()
        outs.append([*fd.values(), press, dt])
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    ctx.close()
