"""The transport path (batches of 750,000 cells and more) with what else a run may ask for: the
learned Newton start, the Riemann stage's block sizes and persistent launch, CUDA graphs, cell
widths that differ along the sweep, and the bounded wait of its TMA tiles."""
import numpy as np
import pytest

import oracle as O
from ppm_b200 import capi
from ppm_b200 import harness as H
from ppm_b200 import learned as LRN
from parity_util import compare, copy_fields, random_state

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    t.cuda.set_device(0)
    return t


SHAPES = [(40, 36, 44), (20, 64, 32), (33, 35, 37), (64, 24, 24)] * 4


def _level(torch, hp):
    grids = [H.Grid.uniform(s) for s in SHAPES]
    assert sum(g.size for g in grids) > 750000 > max(g.size for g in grids)
    host = [random_state(g, hp, seed=70 + k, mach=2.0) for k, g in enumerate(grids)]
    return grids, host


def _dev(torch, host):
    out = [{k: torch.from_numpy(v.copy()).cuda() for k, v in f.items()} for f in host]
    torch.cuda.synchronize()
    return out


@pytest.fixture(scope="module")
def singles(torch):
    """Fields and folded time steps of the level's grids solved one at a time (the separate
    kernels), by build and learned mode."""
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    done = {}

    def get(variant, learned):
        if (variant, learned) not in done:
            grids, host = _level(torch, hp)
            fs = _dev(torch, host)
            c = capi.Context(0, variant=variant)
            c.set_guess(LRN.default_weights())
            dt = torch.full((1,), 1e-3, dtype=torch.float64, device="cuda")
            nxt = torch.zeros(1, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            c.set_cfl(nxt, courant=hp.cfl)
            steps = []
            for cyc in range(3):
                low = []
                for k, g in enumerate(grids):
                    c.solve_ppm_de(g, hp, 0.0, cyc, fs[k], memory=capi.MEM_DEVICE,
                                   learned_guess=learned, dt_device=dt)
                    low.append(nxt.item())
                    c.set_boundary(g, fs[k], True)
                steps.append(min(low))
            assert c.synchronize()[0] == capi.OK
            c.close()
            done[variant, learned] = (fs, steps)
        return done[variant, learned]

    return get


@pytest.mark.parametrize("variant", ["exact", "fast"])
@pytest.mark.parametrize("learned,threads,persistent,graphs", [
    (0, 64, 0, False), (0, 256, 0, False), (0, 64, 1, False), (0, 128, 1, False),
    (0, 256, 1, True), (0, 128, 0, True), (1, 128, 0, False), (2, 128, 0, False),
    (2, 128, 0, True)])
def test_level_options(torch, singles, variant, learned, threads, persistent, graphs):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    ref, steps = singles(variant, learned)
    grids, host = _level(torch, hp)
    fs = _dev(torch, host)
    c = capi.Context(0, variant=variant)
    c.set_guess(LRN.default_weights())
    c.set_graphs(graphs)
    c.set_level_config(riemann_threads=threads, persistent=persistent)
    dt = torch.full((1,), 1e-3, dtype=torch.float64, device="cuda")
    nxt = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    c.set_cfl(nxt, courant=hp.cfl)
    for replay in range(2 if graphs else 1):
        for f, h in zip(fs, host):
            for k in f:
                f[k].copy_(torch.from_numpy(h[k]))
        torch.cuda.synchronize()
        for cyc in range(3):
            c.solve_level(grids, hp, 0.0, cyc, fs, dt_device=dt, learned_guess=learned)
            assert c.synchronize()[0] == capi.OK
            assert nxt.item() == steps[cyc]
            c.set_boundary_level(grids, fs, True)
        assert c.synchronize()[0] == capi.OK
        for a, b in zip(fs, ref):
            for k in a:
                assert torch.equal(a[k], b[k]), (replay, k)
    c.close()


@pytest.mark.parametrize("shape", [(92,) * 3, (95,) * 3])  # TMA tiles, and plain loads
@pytest.mark.parametrize("mode", [1, 2])
def test_learned_start_of_a_single_grid(torch, shape, mode):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    g = H.Grid.uniform(shape)
    f = H.turbulence(g, hp, mach=3.0, seed=31)
    c = capi.Context(0)
    c.set_guess(LRN.default_weights())
    a, b = copy_fields(f), copy_fields(f)
    dt = hp.cfl * O.calc_dt(g, hp, f, O.compute_pressure(g, hp, f), g.cellwidth)
    rc, st_o = O.solve_ppm_de(g, hp, dt, 1, b, g.cellwidth, nthreads=8)
    assert rc == 0
    rc, st = c.solve_ppm_de(g, hp, dt, 1, a, learned_guess=mode)
    assert st["interfaces"] == st_o["interfaces"]
    assert st["newton_iters"] < st_o["newton_iters"]
    for k, r in compare(a, b, g).items():
        assert r["maxrel"] <= 1e-12, (k, r)
    c.close()


# without the filter (it needs one cell width): every active cell's calc_dt
@pytest.mark.parametrize("variant", ["exact", "fast"])
def test_folded_time_step_with_uneven_widths(torch, variant):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.3, dual=True)
    g = H.Grid.uniform((96, 92, 94))
    rng = np.random.default_rng(2)
    w = tuple(np.ascontiguousarray(c * (1.0 + 0.2 * rng.random(c.size))) for c in g.cellwidth)
    g = H.Grid(g.rank, g.dims, g.start, g.end, w)
    f = random_state(g, hp, seed=3)
    f["te"][:, :, 2] += 99.0 * f["ge"][:, :, 2]  # the fastest gas in a ghost plane
    f["ge"][:, :, 2] *= 100.0
    c = capi.Context(0, variant=variant)
    nxt = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    c.set_cfl(nxt, courant=hp.cfl)
    for cyc in range(3):
        fd = _dev(torch, [f])[0]
        c.solve_ppm_de(g, hp, 1e-6, cyc, fd, memory=capi.MEM_DEVICE)
        assert nxt.item() == c.compute_timestep(g, hp, fd, memory=capi.MEM_DEVICE), cyc
    c.close()


# every TMA chunk expects more bytes than its copies deliver, so its barrier never completes:
# each warp gives up after about a second, drains and returns, and the call says so
def test_stalled_tma_waits_time_out_and_the_context_recovers():
    c = capi.Context(0)
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    g = H.Grid.uniform((96, 90, 98))
    f = random_state(g, hp, seed=4)
    dt = hp.cfl * O.calc_dt(g, hp, f, O.compute_pressure(g, hp, f), g.cellwidth)
    try:
        c.debug_tma_stall(16)
        rc, _ = c.solve_ppm_de(g, hp, dt, 0, copy_fields(f), check=False)
        assert rc == capi.ERR_TIMEOUT
    finally:
        c.debug_tma_stall(0)
    a, b = copy_fields(f), copy_fields(f)
    rc, _ = c.solve_ppm_de(g, hp, dt, 0, a)
    assert O.solve_ppm_de(g, hp, dt, 0, b, g.cellwidth, nthreads=8)[0] == 0
    for k, r in compare(a, b, g).items():
        assert r["bitexact"], (k, r)
    c.close()
