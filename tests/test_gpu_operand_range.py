"""The tolerance build over the exponent range of the exact one: its shared reciprocals and
products must stay within the range of a double where the reference's own expressions do.
Those square the differences of a field (the parabola's monotonicity test) and take the third
power of sqrt(gamma*p*d) (the Newton update)."""
import numpy as np
import pytest

from ppm_b200 import capi
from ppm_b200 import harness as H
from parity_util import random_state

pytestmark = pytest.mark.gpu


def _steps(torch, variant, g, hp, p2, d2):
    """Fields after two steps from a state scaled by 2**p2 in pressure and 2**d2 in density
    (velocities by the root of the quotient), scaled back."""
    f = random_state(g, hp, seed=3)
    rng = np.random.default_rng(1)
    v = 2.0 ** ((p2 - d2) // 2)
    unit = {"d": 2.0 ** d2, "v1": v, "v2": v, "v3": v, "te": v * v, "ge": v * v}
    fd = {k: torch.from_numpy(x * unit[k]).cuda() for k, x in f.items()}
    acc = [torch.from_numpy(0.1 * v * v * rng.standard_normal(g.shape)).cuda()
           for _ in range(g.rank)] if hp.gravity else None
    dt = 0.3 / max(g.dims) / 8.0 / v
    c = capi.Context(0, variant=variant)
    for cyc in range(2):
        rc, _ = c.solve_ppm_de(g, hp, dt, cyc, fd, memory=capi.MEM_DEVICE, accel=acc)
        assert rc == capi.OK
    c.close()
    return {k: x.cpu().numpy() / unit[k] for k, x in fd.items()}


# gamma*p*d, the pressure and the density near the largest values in turn; with (100, 480) the
# reference's floors (1e-20 on squared speeds) are active.  Small and transport batches.
@pytest.mark.parametrize("p2,d2,grav", [(0, 0, True), (300, 260, False), (300, 260, True),
                                        (490, -50, True), (100, 480, False)])
@pytest.mark.parametrize("shape,dual", [((40, 24), True), ((40, 24), False), ((900, 900), True)])
def test_tolerance_build_keeps_the_exponent_range(p2, d2, grav, shape, dual):
    torch = pytest.importorskip("torch")
    hp = H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=dual, gravity=grav)
    g = H.Grid.uniform(shape)
    ref = _steps(torch, "exact", g, hp, p2, d2)
    for k, x in _steps(torch, "fast", g, hp, p2, d2).items():
        assert np.isfinite(ref[k]).all() and np.isfinite(x).all(), k
        assert np.abs(x - ref[k]).max() <= 2e-12 * max(np.abs(ref[k]).max(), 1e-300), k
