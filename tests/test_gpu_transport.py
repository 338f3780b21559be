"""The transport path (batches of 750,000 cells and more: v/w/ge reconstruction, fluxes and
update in one kernel) gives the oracle's fields and subgrid fluxes bit for bit, and in the
tolerance build the same bits as the separate kernels that smaller batches run."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from ppm_b200 import capi
from ppm_b200 import harness as H
from parity_util import compare, copy_fields, random_state

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = capi.Context(0)
    yield c
    c.close()


def _check(ctx, g, hp, f, accel=None, cycles=(0, 1, 2), **kw):
    f_gpu, f_ora = copy_fields(f), copy_fields(f)
    for cyc in cycles:
        dt = hp.cfl * O.calc_dt(g, hp, f, O.compute_pressure(g, hp, f), g.cellwidth)
        rc, st_o = O.solve_ppm_de(g, hp, dt, cyc, f_ora, g.cellwidth, accel=accel, nthreads=8)
        assert rc == 0
        rc, st_g = ctx.solve_ppm_de(g, hp, dt, cyc, f_gpu, accel=accel, **kw)
        for key in ("interfaces", "newton_iters", "fallbacks"):
            assert st_g[key] == st_o[key], key
        for k, r in compare(f_gpu, f_ora, g).items():
            assert r["bitexact"], (cyc, k, r)
        H.fill_ghosts(g, f_ora, "periodic")
        H.fill_ghosts(g, f_gpu, "periodic")
    return st_g


# even and odd sides (TMA tiles and plain loads in the x sweep), short and long pencils,
# two dimensions
@pytest.mark.parametrize("shape,dual,grav", [
    ((96, 90, 98), True, False), ((91, 93, 95), True, True), ((96, 96, 90), False, True),
    ((900, 901), True, False), ((1001, 760), False, False), ((2, 330, 331), True, False),
    ((330, 4, 330), True, False)])
def test_transport_matches_oracle(ctx, shape, dual, grav):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=dual, gravity=grav)
    g = H.Grid.uniform(shape)
    rng = np.random.default_rng(4)
    accel = [0.1 * rng.standard_normal(g.shape) for _ in range(g.rank)] if grav else None
    _check(ctx, g, hp, random_state(g, hp, seed=sum(shape)), accel,
           cycles=(0, 1, 2)[:g.rank])


@pytest.mark.parametrize("flatten,steepen", [(3, 1), (1, 0), (0, 1)])
def test_transport_with_slope_corrections(ctx, flatten, steepen):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True, flatten=flatten, steepen=steepen)
    g = H.Grid.uniform((94, 90, 96))
    _check(ctx, g, hp, random_state(g, hp, seed=8, mach=3.0), cycles=(1,))


def test_transport_with_uneven_widths(ctx):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.3, dual=True)
    g = H.Grid.uniform((96, 92, 94))
    rng = np.random.default_rng(2)
    w = tuple(np.ascontiguousarray(c * (1.0 + 0.2 * rng.random(c.size))) for c in g.cellwidth)
    g = H.Grid(g.rank, g.dims, g.start, g.end, w)
    _check(ctx, g, hp, random_state(g, hp, seed=3), cycles=(0,))


# flagged pencils get their advected states and fluxes in the fallback pass
@pytest.mark.parametrize("shape", [(96, 90, 98), (95, 93, 96)])
def test_transport_fallback(ctx, shape):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    g = H.Grid.uniform(shape)
    f = random_state(g, hp, seed=6, mach=0.3)
    rng = np.random.default_rng(1)
    for _ in range(40):
        k, j, i = (int(rng.integers(3, n - 3)) for n in g.shape)
        f["te"][k, j, i] = -1e-3
    dt = 1e-4
    f_gpu, f_ora = copy_fields(f), copy_fields(f)
    rc, st_o = O.solve_ppm_de(g, hp, dt, 0, f_ora, g.cellwidth, nthreads=8)
    assert rc == 0 and st_o["fallbacks"] >= 40
    rc, st_g = ctx.solve_ppm_de(g, hp, dt, 0, f_gpu)
    assert st_g["fallbacks"] == st_o["fallbacks"]
    for k, r in compare(f_gpu, f_ora, g).items():
        assert r["bitexact"], (k, r)


def test_transport_subgrid_fluxes(ctx):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    g = H.Grid.uniform((96, 94, 90))
    f = random_state(g, hp, seed=12)
    lo, hi = (3, 30, 17), (98, 61, 80)  # the left face of the grid itself, and its right one

    def box():
        b = {k: [[0] * 3 for _ in range(3)]
             for k in ("left_start", "left_end", "right_start", "right_end")}
        b["left"] = [[None] * 3 for _ in range(6)]
        b["right"] = [[None] * 3 for _ in range(6)]
        for d in range(3):
            for j in range(3):
                b["left_start"][d][j], b["left_end"][d][j] = lo[j], hi[j] if j != d else lo[j]
                b["right_start"][d][j], b["right_end"][d][j] = lo[j] if j != d else hi[j], hi[j]
            n = int(np.prod([hi[j] - lo[j] + 1 for j in range(3) if j != d]))
            for s in range(6):
                b["left"][s][d], b["right"][s][d] = np.zeros(n), np.zeros(n)
        return b

    bg, bo = box(), box()
    of = O.OraFluxes()
    for key in ("left_start", "left_end", "right_start", "right_end"):
        for i in range(3):
            for j in range(3):
                getattr(of, key)[i][j] = bo[key][i][j]
    for side in ("left", "right"):
        for s in range(6):
            for d in range(3):
                getattr(of, side)[s][d] = bo[side][s][d].ctypes.data_as(C.POINTER(C.c_double))
    f_gpu, f_ora = copy_fields(f), copy_fields(f)
    rc, _ = O.solve_ppm_de(g, hp, 1e-4, 0, f_ora, g.cellwidth, subgrids=[of], ggs=(0, 0, 0))
    assert rc == 0
    ctx.solve_ppm_de(g, hp, 1e-4, 0, f_gpu, subgrids=[bg])
    for side in ("left", "right"):
        for s in range(6):
            for d in range(3):
                assert np.array_equal(bg[side][s][d], bo[side][s][d]), (side, s, d)


@pytest.mark.parametrize("variant", ["exact", "fast"])
@pytest.mark.parametrize("dual,grav", [(True, False), (False, False), (True, True)])
def test_level_batch_and_single_grids_take_both_paths(variant, dual, grav):
    torch = pytest.importorskip("torch")
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=dual, gravity=grav)
    shapes = [(40, 36, 44), (20, 64, 32), (33, 35, 37), (64, 24, 24)] * 4
    grids = [H.Grid.uniform(s) for s in shapes]
    assert sum(g.size for g in grids) > 750000 > max(g.size for g in grids)
    host = [random_state(g, hp, seed=40 + k) for k, g in enumerate(grids)]
    rng = np.random.default_rng(3)
    acc = [[torch.from_numpy(0.1 * rng.standard_normal(g.shape)).cuda() for _ in range(3)]
           if grav else None for g in grids]
    dev = lambda: [{k: torch.from_numpy(v.copy()).cuda() for k, v in f.items()}  # noqa: E731
                   for f in host]
    one, batch = dev(), dev()
    c = capi.Context(0, variant=variant)
    dts = [torch.zeros(1, dtype=torch.float64, device="cuda") for _ in grids]
    dt_batch = torch.zeros(1, dtype=torch.float64, device="cuda")
    for cyc in range(3):
        for k, g in enumerate(grids):
            c.set_cfl(dts[k], courant=hp.cfl)
            c.solve_ppm_de(g, hp, 1e-3, cyc, one[k], memory=capi.MEM_DEVICE, accel=acc[k],
                           want_stats=False)
        c.set_cfl(dt_batch, courant=hp.cfl)
        c.solve_level(grids, hp, 1e-3, cyc, batch, accels=acc if grav else None)
        assert c.synchronize()[0] == capi.OK
        assert dt_batch.item() == min(d.item() for d in dts)
        for k, g in enumerate(grids):
            for n in one[k]:
                assert torch.equal(one[k][n], batch[k][n]), (cyc, k, n)
            c.set_boundary(g, one[k], dual)
        c.set_boundary_level(grids, batch, dual)
    c.set_cfl(None)
    c.close()
