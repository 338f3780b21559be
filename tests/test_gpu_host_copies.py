"""Host-memory calls: pageable fields go through the context's pinned pieces (threads above
4 MB a call), pinned fields directly; the fields are the device call's either way."""
import resource
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from ppm_b200 import capi
from ppm_b200 import harness as H
from parity_util import copy_fields, random_state

pytestmark = pytest.mark.gpu


# below and above the size worth the threads, pieces with ragged ends, more than the staging
# memory holds at once (64 MiB), colours
@pytest.mark.parametrize("shape,ncol", [((20, 18, 16), 0), ((40, 41, 43), 0), ((64, 64, 64), 3),
                                        ((120, 121, 122), 0)])
@pytest.mark.parametrize("grav", [False, True])
def test_pageable_pinned_and_device_fields_agree(shape, ncol, grav):
    torch = pytest.importorskip("torch")
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True, gravity=grav)
    g = H.Grid.uniform(shape)
    f = random_state(g, hp, seed=4)
    rng = np.random.default_rng(1)
    for n in range(ncol):
        f[f"col{n}"] = f["d"] * (0.1 + rng.random(g.shape))
    acc = [0.1 * rng.standard_normal(g.shape) for _ in range(3)] if grav else None
    c = capi.Context(0)
    dev = {k: torch.from_numpy(v).cuda() for k, v in f.items()}
    acc_dev = [torch.from_numpy(a).cuda() for a in acc] if grav else None
    host = {k: v.copy() for k, v in f.items()}
    pinned = {k: torch.from_numpy(v.copy()).pin_memory() for k, v in f.items()}
    pinned_np = {k: v.numpy() for k, v in pinned.items()}
    for cyc in range(2):
        c.solve_ppm_de(g, hp, 1e-3, cyc, dev, memory=capi.MEM_DEVICE, accel=acc_dev)
        c.solve_ppm_de(g, hp, 1e-3, cyc, host, accel=acc)
        c.solve_ppm_de(g, hp, 1e-3, cyc, pinned_np, accel=acc)
        for k in f:
            ref = dev[k].cpu().numpy()
            assert np.array_equal(host[k], ref), (cyc, k)
            assert np.array_equal(pinned_np[k], ref), (cyc, k)
    c.close()


# calls that only read the fields: the driver's copies up to a larger size, then the pieces
@pytest.mark.parametrize("shape", [(40, 41, 43), (64, 64, 64), (90, 91, 92)])
def test_calls_that_only_read_host_fields(shape):
    torch = pytest.importorskip("torch")
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    g = H.Grid.uniform(shape)
    f = random_state(g, hp, seed=4)
    dev = {k: torch.from_numpy(v).cuda() for k, v in f.items()}
    c = capi.Context(0)
    p, pd = np.zeros(g.shape), torch.zeros(g.shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        assert c.compute_timestep(g, hp, f) == c.compute_timestep(g, hp, dev,
                                                                  memory=capi.MEM_DEVICE)
        c.compute_pressure(g, hp, f, p)
        c.compute_pressure(g, hp, dev, pd, memory=capi.MEM_DEVICE)
        torch.cuda.synchronize()
        assert np.array_equal(p, pd.cpu().numpy())
    c.close()


# a context on a stream of the caller's: the legacy and the per-thread default stream (whose
# handles, 1 and 2, name the calling thread's own stream) and a created one
@pytest.mark.parametrize("stream", [1, 2, "created"])
def test_host_fields_on_the_callers_stream(stream):
    torch = pytest.importorskip("torch")
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    g = H.Grid.uniform((64, 64, 64))
    f = random_state(g, hp, seed=4)
    own = torch.cuda.Stream()
    ref, ctx = capi.Context(0), capi.Context(0, stream=own.cuda_stream if stream == "created"
                                             else stream)
    a, b = copy_fields(f), copy_fields(f)
    for cyc in range(3):
        ref.solve_ppm_de(g, hp, 1e-3, cyc, a)
        ctx.solve_ppm_de(g, hp, 1e-3, cyc, b)
        for k in f:
            assert np.array_equal(a[k], b[k]), (cyc, k)
    ctx.close()
    ref.close()


# No pinned memory to be had (the process's address space is full): the call takes the
# driver's copies.  In a process of its own.
def no_pinned_memory():
    import torch

    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    g = H.Grid.uniform((64, 64, 64))
    f = random_state(g, hp, seed=4)
    c = capi.Context(0)
    pinned = {k: torch.from_numpy(v.copy()).pin_memory() for k, v in f.items()}
    ref = {k: v.numpy() for k, v in pinned.items()}
    c.solve_ppm_de(g, hp, 1e-3, 0, ref)  # allocates all the call needs but the staging
    used = int(Path("/proc/self/statm").read_text().split()[0]) * resource.getpagesize()
    soft, hard = resource.getrlimit(resource.RLIMIT_AS)
    resource.setrlimit(resource.RLIMIT_AS, (used + (1 << 20), hard))
    rc, _ = c.solve_ppm_de(g, hp, 1e-3, 0, f, check=False)
    resource.setrlimit(resource.RLIMIT_AS, (soft, hard))
    assert rc == capi.OK
    for k in f:
        assert np.array_equal(f[k], ref[k]), k
    c.close()


def test_no_pinned_memory():
    here = Path(__file__).resolve().parent
    code = (f"import sys; sys.path[:0] = [{str(here)!r}, {str(here.parent / 'enzo-dev_b200')!r}]; "
            "import test_gpu_host_copies as t; t.no_pinned_memory()")
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300)
