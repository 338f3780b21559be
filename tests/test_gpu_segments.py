"""The marching stages cut long pencils into segments when a batch has few of them
(set_segments): every split gives the oracle's fields bit for bit, like whole pencils."""
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


def _steps(ctx, g, hp, f, cycles=3, plant=None):
    f_gpu, f_ora = copy_fields(f), copy_fields(f)
    for cyc in range(cycles):
        if plant and cyc == 0:
            for a in (f_gpu, f_ora):
                for idx in plant:
                    a["te"][idx] = -1e-3
        dt = hp.cfl * O.calc_dt(g, hp, f, O.compute_pressure(g, hp, f), g.cellwidth)
        rc, st_o = O.solve_ppm_de(g, hp, dt, cyc, f_ora, g.cellwidth)
        assert rc == 0
        rc, st_g = ctx.solve_ppm_de(g, hp, dt, cyc, f_gpu)
        assert st_g["fallbacks"] == st_o["fallbacks"]
        for k, r in compare(f_gpu, f_ora, g).items():
            assert r["bitexact"], (cyc, k, r)
        H.fill_ghosts(g, f_ora, "periodic")
        H.fill_ghosts(g, f_gpu, "periodic")


# segments of 4 faces up to the whole pencil: shorter than a segment, just above the split
# points, ragged last segments, pencils per block from 1 to 128
@pytest.mark.parametrize("shape", [(2,), (6,), (7,), (8,), (15,), (61,), (124,), (1000,),
                                   (8, 3), (33, 130), (127, 40, 3), (5, 64, 64)])
@pytest.mark.parametrize("dual", [True, False])
def test_every_split_matches_oracle(ctx, shape, dual):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=dual)
    g = H.Grid.uniform(shape)
    _steps(ctx, g, hp, random_state(g, hp, seed=sum(shape)))


# a bad cell anywhere in a pencil hands all its segments to the fallback pass, once
@pytest.mark.parametrize("cells", [(3,), (6,), (7,), (10, 11), (3, 40, 41, 66), (66,)])
def test_fallback_reaches_every_segment_of_its_pencil(ctx, cells):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True)
    g = H.Grid.uniform((64, 6))
    f = random_state(g, hp, seed=5, mach=0.3)
    _steps(ctx, g, hp, f, cycles=1, plant=[(0, 5, i) for i in cells])


# eta1 > eta2/4: a cell's energy may depend on its left neighbour's, so the pencils stay
# whole; eta1 = eta2/4: the last value that splits; cold gas takes both branches
@pytest.mark.parametrize("eta1,eta2", [(0.2, 0.1), (0.025, 0.1), (0.0251, 0.1), (0.0, 0.0)])
def test_dual_energy_select_parameters(ctx, eta1, eta2):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True, eta1=eta1, eta2=eta2)
    g = H.Grid.uniform((70, 12))
    _steps(ctx, g, hp, random_state(g, hp, seed=9, mach=8.0))


# a negative eta2: an internal energy below zero passes the test beside a neighbour of larger
# energy where it would not by itself, so the pencils stay whole
@pytest.mark.parametrize("seed,eta1,eta2", [(3, -0.3, -0.3), (5, -1.0, -1.0), (8, -0.3, -0.3),
                                            (12, -2.0, -0.6)])
def test_dual_energy_select_of_negative_thresholds(ctx, seed, eta1, eta2):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.1, dual=True, eta1=eta1, eta2=eta2)
    g = H.Grid.uniform((1000,))
    f = random_state(g, hp, seed=seed, mach=8.0)
    rng = np.random.default_rng(seed)
    low = rng.random(g.shape) < 0.6
    f["te"][low] = (0.5 * f["v1"] ** 2 * rng.uniform(0.1, 0.7, g.shape))[low]
    _steps(ctx, g, hp, f, cycles=1)


# colours are updated in place by the segments of a pencil; flattening and steepening
# coefficients come in the same split
@pytest.mark.parametrize("shape,ncol", [((9,), 1), ((130,), 3), ((40, 37), 2), ((17, 33, 20), 5)])
@pytest.mark.parametrize("flatten,steepen", [(0, 0), (3, 1)])
def test_colours_in_segments(ctx, shape, ncol, flatten, steepen):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=True, flatten=flatten, steepen=steepen)
    g = H.Grid.uniform(shape)
    f = random_state(g, hp, seed=11)
    rng = np.random.default_rng(12)
    for n in range(ncol):
        f[f"col{n}"] = f["d"] * (0.2 + 0.5 * rng.random(g.shape))
    H.fill_ghosts(g, f, "periodic")
    _steps(ctx, g, hp, f)


# cell widths that differ along the sweep take the general reconstruction
def test_uneven_cell_widths(ctx):
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.3, dual=True)
    g = H.Grid.uniform((40, 14))
    rng = np.random.default_rng(2)
    w = [np.ascontiguousarray(c * (1.0 + 0.2 * rng.random(c.size))) if c.size > 1 else c
         for c in g.cellwidth]
    g = H.Grid(g.rank, g.dims, g.start, g.end, tuple(w))
    _steps(ctx, g, hp, random_state(g, hp, seed=3))
