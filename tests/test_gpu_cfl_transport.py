"""The folded time step (ppm_b200_set_cfl) on the transport path (batches of 750,000 cells and
more): equal to the separate calc_dt pass, whose cells are the active ones alone -- with the
fastest gas of the batch in the ghost planes beside the grid, and with pencils that the last
sweep hands to the fallback pass."""
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


# gas 100 times as hot (10 times the signal speed) in the planes next to the active cells; over
# a step of 1e-6 no active cell gets near it
DT = 1e-6


def _heat_ghosts(g, f, hp):
    axes = {0: 2, 1: 1, 2: 0}  # array axis of x, y, z
    hot = np.zeros(g.shape, dtype=bool)
    for d in range(g.rank):
        for i in (g.start[d] - 1, g.end[d] + 1):
            idx = [slice(None)] * 3
            idx[axes[d]] = i
            hot[tuple(idx)] = True
    ke = 0.5 * sum(f[v] ** 2 for v in ("v1", "v2", "v3")[:g.rank])
    eint = f["te"] - ke
    f["te"][hot] = (100.0 * eint + ke)[hot]
    if hp.dual:
        f["ge"][hot] = 100.0 * eint[hot]


# cells with a negative total energy; without the dual-energy select they keep it through
# every sweep of a step this small, so the last sweep flags their pencils too
def _bad_cells(g, f, torch, n=30):
    gen = torch.Generator().manual_seed(n)
    for _ in range(n):
        k, j, i = (int(torch.randint(3, s - 3, (1,), generator=gen)) if s > 6 else 0
                   for s in g.shape)
        f["te"][k, j, i] = -1.0
    return int((f["te"] == -1.0).sum())


# even and odd sides (TMA tiles and the ring in the x sweep), two dimensions; every sweep last
@pytest.mark.parametrize("variant", ["exact", "fast"])
@pytest.mark.parametrize("shape", [(96, 90, 98), (91, 93, 95), (900, 901)])
@pytest.mark.parametrize("dual,bad", [(True, False), (False, False), (False, True)])
def test_single_grid(torch, variant, shape, dual, bad):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.45, dual=dual)
    g = H.Grid.uniform(shape, width=tuple(0.7 + 0.2 * d for d in range(len(shape))))
    assert g.size >= 750000
    f = random_state(g, hp, seed=sum(shape), mach=0.5)
    _heat_ghosts(g, f, hp)
    n = _bad_cells(g, f, torch) if bad else 0
    ctx = capi.Context(0, variant=variant)
    nxt = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    kw = dict(aye=0.9, vgrid=(0.01, -0.02, 0.03))
    ctx.set_cfl(nxt, courant=hp.cfl, **kw)
    for cyc in range(g.rank):
        fd = {k: torch.from_numpy(v.copy()).cuda() for k, v in f.items()}
        rc, st = ctx.solve_ppm_de(g, hp, DT, cyc, fd, memory=capi.MEM_DEVICE)
        assert st["fallbacks"] >= n * g.rank  # n in each sweep
        ref = ctx.compute_timestep(g, hp, fd, memory=capi.MEM_DEVICE, **kw)
        assert nxt.item() == ref, (cyc, nxt.item(), ref)
    ctx.close()


@pytest.mark.parametrize("variant", ["exact", "fast"])
@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("dual,bad", [(True, False), (False, True)])
def test_level(torch, variant, graphs, dual, bad):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=dual)
    shapes = [(40, 36, 44), (20, 64, 32), (33, 35, 37), (64, 24, 24), (16, 16, 16)] * 4
    grids = [H.Grid.uniform(s) for s in shapes]
    assert sum(g.size for g in grids) >= 750000
    host = [random_state(g, hp, seed=60 + k, mach=0.5) for k, g in enumerate(grids)]
    n = 0
    for g, f in zip(grids, host):
        _heat_ghosts(g, f, hp)
        n += _bad_cells(g, f, torch, n=3) if bad else 0
    ctx = capi.Context(0, variant=variant)
    ctx.set_graphs(graphs)
    dt = torch.zeros(1, dtype=torch.float64, device="cuda")
    nxt = torch.zeros(1, dtype=torch.float64, device="cuda")
    dt.fill_(DT)
    torch.cuda.synchronize()
    ctx.set_cfl(nxt, courant=hp.cfl)
    fs = [{k: torch.empty(v.shape, dtype=torch.float64, device="cuda") for k, v in f.items()}
          for f in host]
    for cyc in (0, 1, 2, 0, 1, 2):  # the second time round replays
        for f, h in zip(fs, host):
            for k in f:
                f[k].copy_(torch.from_numpy(h[k]))
        torch.cuda.synchronize()
        rc, st = ctx.solve_level(grids, hp, 0.0, cyc, fs, dt_device=dt, want_stats=True)
        assert st["fallbacks"] >= 3 * n
        ref = ctx.compute_timestep_level(grids, hp, fs)
        assert nxt.item() == ref, (cyc, nxt.item(), ref)
    ctx.close()


# without a pressure floor a cold cell's pressure is zero (its total energy less than its
# kinetic one after the step): it still moves, and may be the fastest
@pytest.mark.parametrize("variant", ["exact", "fast"])
def test_cells_without_pressure(torch, variant):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=False, tiny_number=0.0)
    g = H.Grid.uniform((900, 900))
    f = random_state(g, hp, seed=2, mach=1e4)
    ctx = capi.Context(0, variant=variant)
    nxt = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.set_cfl(nxt, courant=hp.cfl)
    fd = {k: torch.from_numpy(v.copy()).cuda() for k, v in f.items()}
    dt = ctx.compute_timestep(g, hp, fd, memory=capi.MEM_DEVICE)
    rc, _ = ctx.solve_ppm_de(g, hp, dt, 0, fd, memory=capi.MEM_DEVICE, check=False)
    assert rc in (capi.OK, capi.ERR_NEGATIVE)
    cold = fd["te"] - 0.5 * (fd["v1"] ** 2 + fd["v2"] ** 2) <= 0.0
    assert int(cold[0, 3:-3, 3:-3].sum()) > 1000
    assert nxt.item() == ctx.compute_timestep(g, hp, fd, memory=capi.MEM_DEVICE)
    ctx.close()
