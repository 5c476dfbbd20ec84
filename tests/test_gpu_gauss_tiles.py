"""The Gauss pass in tiles, where blocks share out the planes of all tiles (GPU).

Every local violation and the rows against the oracle's FP64 Gauss pass over the very fields the
step left, widened exactly to double: lattices whose edges leave tiles ragged in y and z, whose planes
do not share out evenly, with and without Fixed
faces.  Bars as derived in test_gpu_tiled.py: 1e-12 of the maximum and the integral; one float
ulp plus 1e-16 of each local violation.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,shape,fixed", [
    (1, (1, 683, 448), 0),    # one plane: each its own back neighbour, a march begins every plane
    (1, (3, 338, 300), 7),    # 48.3 tiles along y, 9.4 along z
    (1, (107, 54, 54), 0),    # shares of five or six planes from one tile's end into the next
    (2, (107, 54, 54), 5),
    (2, (2, 470, 320), 0),
])
def test_gauss_in_tiles_matches_oracle_on_the_same_fields(oracle_mod, model, shape, fixed):
    from gftevolver_b200 import Evolver, LatticeParams
    nx, ny, nz = shape
    op = oracle_mod.Params(model=model, nx=nx, ny=ny, nz=nz, gauss_every=1, gauss_local_every=1, fixed_axes=fixed)
    ic = oracle_mod.ICSpec(seed=43, mean=[1.0 if model == 1 else 0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1,
                           eps_sigma=0.1)
    sc, ve = oracle_mod.init_fields(op, ic, np.float32)
    with Evolver(LatticeParams(**op.__dict__), form="mixed") as ev:
        ev.upload(sc, ve, 0)
        rows = ev.evolve(3)
        g_sc, g_ve = ev.download()
        _, _, lg, _ = ev.local_fields()
    gi, gm, o_lg = oracle_mod.gauss(op, g_sc.astype(np.float64), g_ve.astype(np.float64), 2)
    np.testing.assert_allclose(rows[-1]["gauss_max"], gm, rtol=1e-12, atol=1e-18)
    np.testing.assert_allclose(rows[-1]["gauss_int"], gi, rtol=1e-12, atol=1e-18)
    tol = np.spacing(np.abs(o_lg).astype(np.float32)).astype(np.float64) + 1e-16
    assert (np.abs(lg.astype(np.float64) - o_lg) - tol).max() <= 0.0


@pytest.mark.parametrize("model", [1, 2])
def test_ensemble_gauss_rows_match_oracle_on_the_same_fields(oracle_mod, model):
    """Members whose Gauss pass runs in tiles and by single sites (nz = 16) in one batch: the last
    row of each against the oracle on that member's fields, as above."""
    from gftevolver_b200 import Ensemble, InitialData, LatticeParams
    shapes = [(20, 16, 16), (9, 28, 32), (40, 44, 48), (5, 8, 64), (64, 64, 64)]
    ops = [oracle_mod.Params(model=model, nx=a, ny=b, nz=c, gauss_every=2) for a, b, c in shapes]
    with Ensemble([LatticeParams(**op.__dict__) for op in ops]) as ens:
        ens.init_fields([InitialData(seed=7 + m, mean=[0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1, eps_sigma=0.1)
                         for m in range(len(ops))])
        rows = ens.evolve(5)
        fields = [ens.download(m) for m in range(len(ops))]
    for op, got, (sc, ve) in zip(ops, rows, fields):
        assert got[-1]["time_iter"] == 4 and got[-1]["has_gauss"]
        gi, gm, _ = oracle_mod.gauss(op, sc.astype(np.float64), ve.astype(np.float64), 4)
        np.testing.assert_allclose(got[-1]["gauss_max"], gm, rtol=1e-12, atol=1e-18)
        np.testing.assert_allclose(got[-1]["gauss_int"], gi, rtol=1e-12, atol=1e-18)
