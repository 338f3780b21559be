"""The next cycle's time step folded into the last sweep (ppm_b200_set_cfl): the value
written by a solve equals the separate calc_dt pass (ppm_b200_compute_timestep) on the
updated fields bit for bit -- single grids of every rank, with and without dual energy
and gravity, with HLL-fallback pencils, levels, and CUDA-graph replays."""
import numpy as np
import pytest

from ppm_b200 import capi
from ppm_b200 import harness as H
from parity_util import random_state

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    t.cuda.set_device(0)
    return t


def _dev(f, torch):
    return {k: torch.from_numpy(v.copy()).cuda() for k, v in f.items()}


@pytest.mark.parametrize("shape,dual,grav,fallback_cells", [
    ((16, 12, 10), True, False, False),
    ((16, 12, 10), False, False, False),
    ((14, 11, 9), True, True, False),
    ((20, 12, 10), True, False, True),
    ((24, 18), True, False, False),
    ((40,), False, False, False),
    # x sweep staged with lanes past the last pencil (72 pencils of 32 a warp), which have no
    # cell widths to read
    ((16, 2, 3), True, False, False),
    ((16, 2, 3), False, True, False),
])
def test_folded_time_step_equals_calc_dt(torch, shape, dual, grav, fallback_cells):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.45, dual=dual, gravity=grav)
    g = H.Grid.uniform(shape, width=tuple(0.5 + 0.1 * d for d in range(len(shape))))
    f = random_state(g, hp, seed=55)
    if fallback_cells:
        for (k, j, i) in [(5, 6, 8), (5, 6, 9), (8, 4, 14)]:
            f["te"][k, j, i] = -1e-3
    accel = None
    if grav:
        rng = np.random.default_rng(5)
        accel = [torch.from_numpy(0.1 * rng.standard_normal(g.shape)).cuda()
                 for _ in range(g.rank)]
    fd = _dev(f, torch)
    ctx = capi.Context(0)
    nxt = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.set_cfl(nxt, courant=hp.cfl, aye=0.9, vgrid=(0.01, -0.02, 0.03))
    for cyc in range(3):
        dt = ctx.compute_timestep(g, hp, fd, memory=capi.MEM_DEVICE, aye=0.9,
                                  vgrid=(0.01, -0.02, 0.03))
        rc, st = ctx.solve_ppm_de(g, hp, dt, cyc, fd, memory=capi.MEM_DEVICE, accel=accel,
                                  check=False)
        assert rc == capi.OK
        if fallback_cells and cyc == 0:
            assert st["fallbacks"] > 0
        ref = ctx.compute_timestep(g, hp, fd, memory=capi.MEM_DEVICE, aye=0.9,
                                   vgrid=(0.01, -0.02, 0.03))
        assert nxt.item() == ref, (cyc, nxt.item(), ref)
        ctx.set_boundary(g, fd, dual)
    ctx.close()


def test_folded_time_step_of_a_level_with_graphs(torch):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    shapes = [(16, 16, 16), (24, 12, 8), (8, 8, 8), (10, 18, 6)]
    grids = [H.Grid.uniform(s) for s in shapes]
    fs = [_dev(random_state(g, hp, seed=100 + k), torch) for k, g in enumerate(grids)]
    ctx = capi.Context(0)
    ctx.set_graphs(True)
    dt = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.compute_timestep_level(grids, hp, fs, dt_device=dt, want_host=False)
    ctx.set_cfl(dt, courant=hp.cfl)
    for cyc in range(5):  # the solve reads dt and leaves the next one in it
        ctx.solve_level(grids, hp, 0.0, cyc, fs, dt_device=dt)
        ref = ctx.compute_timestep_level(grids, hp, fs)
        assert dt.item() == ref, (cyc, dt.item(), ref)
        ctx.set_boundary_level(grids, fs, True)
    ctx.close()


# A pencil cut into segments of eight cells, whose bad cell b (its density runs out along the
# last sweep) lies two cells from a segment border: the fallback changes the energy of cell
# b+1, hence the dual-energy select of cell b+2, which another segment has stored by then with
# the hot gas energy it no longer has.  The signal speed of that state must not keep the true
# fastest cell (another pencil of the block, the last cell of its segment) out of the minimum.
@pytest.mark.parametrize("u,dt,ub,db,dc,dm,de,up", [
    (2.2498, 0.0089198, 0.0, 0.63657, 0.38141, 1.1054, 6.8954, True),
    (1.4972, 0.012593, 0.0, 2.2955, 2.0466, 1.5901, 7.4858, False),
    (1.3202, 0.017501, 0.0, 2.4083, 2.3949, 2.8732, 8.024, False),
    (2.5989, 0.0093248, 0.0, 0.53066, 0.38457, 2.1178, 8.5972, False),
])
@pytest.mark.parametrize("variant", ["exact", "fast"])
def test_folded_time_step_beside_a_flagged_pencil(torch, variant, u, dt, ub, db, dc, dm, de, up):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    g = H.Grid.uniform((20, 64), width=(20 / 64, 1.0))
    bad, hot = 10, 13  # pencils along y
    b, step = (22, 1) if up else (25, -1)
    d, v = np.ones(g.shape), np.full(g.shape, 6.0)
    v[:, :, (bad, hot)] = 0.0
    v[0, b, bad], v[0, b - step, bad] = step * u, step * u * ub
    d[0, b, bad], d[0, b + step, bad], d[0, b - step, bad] = db, dc, dm
    d[0, b + 2 * step, bad] = 0.03
    d[0, 39, hot] = 0.045
    ge = 1.5 / d  # one pressure: nothing moves along x
    te = ge + 0.5 * v ** 2
    te[0, b + 2 * step, bad] = 0.1 * de / 0.03  # the select's threshold between the two
    zero = np.zeros(g.shape)
    f = dict(d=d, te=te, v1=zero, v2=v, v3=zero, ge=ge)
    ctx = capi.Context(0, variant=variant)
    nxt = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.set_cfl(nxt, courant=hp.cfl)
    fd = _dev(f, torch)
    rc, st = ctx.solve_ppm_de(g, hp, dt, 0, fd, memory=capi.MEM_DEVICE)
    assert st["fallbacks"] > 0
    assert fd["ge"][0, b + 2 * step, bad].item() < 30.0  # selected again (50 before)
    assert nxt.item() == ctx.compute_timestep(g, hp, fd, memory=capi.MEM_DEVICE)
    ctx.close()
