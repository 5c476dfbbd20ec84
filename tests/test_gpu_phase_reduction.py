"""The FP64 form's sines next to a multiple of pi (GPU).

91.106186954104 is the double nearest to 29 pi, 1.2e-18 from it.  Phases that turn by twice that a
step, in a vacuum of unit links, leave the electric energy of the phases alone, a sum of 1 - cos =
2 sin^2 of that number, which keeps the sine's relative accuracy.  Bar: 1e-14 of it, the square of a
sine good to some ulp, its reduction by pi included.
"""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PI = Fraction("3.14159265358979323846264338327950288419716939937510582097494459230781640628620899")
NEAR = 91.106186954104


@pytest.mark.parametrize("shape,kind", [((8, 8, 8), 0), ((33, 32, 32), 0), ((4, 24, 96), 2)],
                         ids=["divided", "one_thread_per_site", "tiles"])
@pytest.mark.parametrize("model,family", [(1, 0), (2, 0), (2, 1)])
def test_electric_energy_of_phases_near_a_multiple_of_pi(oracle_mod, model, family, shape, kind):
    from gftevolver_b200 import Evolver, LatticeParams
    if kind and model != 1:
        pytest.skip("the caller's FP64 tiles serve the SM model")
    nx, ny, nz = shape
    op = oracle_mod.Params(model=model, nx=nx, ny=ny, nz=nz, dt=0.25, g=1.0, gp=0.5, gpp=0.5, higgs_family=family,
                           energy_every=1)
    sc, ve = oracle_mod.init_fields(op, oracle_mod.ICSpec(sigma=[0.0] * 8), np.float64)
    dw = ve.shape[-1] // 3
    turning = [0] + ([5] if family else [])
    for d in range(3):
        for at in turning:
            ve[1][..., dw * d + at] = 2 * NEAR  # "now" at time_iter 0; the past phases are zero
    with Evolver(LatticeParams(**op.__dict__), form="fp64") as ev:
        if kind:
            ev.set_kernel(kind, 0, 4)
        ev.upload(sc, ve, 0)
        row = ev.evolve(1)[0]
    sine = float(Fraction(NEAR) - 29 * PI)  # sin r = r (1 - r^2 / 6)
    want = nx * ny * nz * 3 * len(turning) * 4 / 0.25 ** 2 / 0.5 ** 2 * 2 * sine ** 2
    assert want > 0 and abs(row["electric"] / want - 1) <= 1e-14
