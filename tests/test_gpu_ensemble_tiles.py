"""Which tiles an ensemble takes by itself (GPU), told by its energy rows: their partial sums are a
tile's, so another tile's rows differ in their last digits."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,sizes,tile,other", [
    (1, [(16, 16, 16)] * 3, 2, 3),                   # narrow planes: 4 x 16, not one 16 x 16 tile each
    (1, [(16, 16, 48), (40, 48, 16)], 2, 3),
    (1, [(16, 16, 16), (16, 16, 64)], 3, 2),         # one member of more than 768 sites a plane
    (1, [(32, 32, 32)] * 2, 3, 0),
    (2, [(32, 32, 32)] * 2, 0, 3),
])
def test_default_tile(model, sizes, tile, other):
    from gftevolver_b200 import Ensemble, InitialData, LatticeParams
    ps = [LatticeParams(model=model, nx=s[0], ny=s[1], nz=s[2], energy_every=1) for s in sizes]
    ics = [InitialData(seed=5 + m, mean=[1.0 if model == 1 else 0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1, eps_sigma=0.1)
           for m in range(len(sizes))]
    rows = []
    for t in (None, tile, other):
        with Ensemble(ps) as ens:
            if t is not None:
                ens.set_kernel(t, 24)
            ens.init_fields(ics)
            rows.append(ens.evolve(2))
    assert rows[0] == rows[1] != rows[2]
