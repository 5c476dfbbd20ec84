"""The reference-arithmetic step of generator links with five blocks per SM (GPU).

48^3 sites are 1,152 blocks of 32 x 4, a wave of seven per SM and a few more: the step takes the
instance with five.  Plain and logging steps against the oracle, with the bars of the form
(test_gpu_parity.py): 8 float ulps, at most 1 % of the words different, energies to 2e-5; with FP64
storage 1e-13 of the fields, energies to 1e-12.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,dtype", [("ref32", np.float32), ("ref64", np.float64)])
def test_generator_step_of_little_more_than_a_wave(oracle_mod, form, dtype):
    from gftevolver_b200 import Evolver, LatticeParams
    op = oracle_mod.Params(model=1, nx=48, ny=48, nz=48, generator_rep=1, energy_every=2, gauss_every=2)
    ic = oracle_mod.ICSpec(seed=4, mean=[1.0] * 8, sigma=[0.1] * 8, theta_sigma=0.1, eps_sigma=0.1)
    sc, ve = oracle_mod.init_fields(op, ic, dtype)
    with Evolver(LatticeParams(**op.__dict__), form=form) as ev:
        ev.upload(sc, ve, 0)
        rows = ev.evolve(3)
        assert ev.last_warnings == 0
        got = ev.download()
    o_rows, _ = oracle_mod.evolve(op, sc, ve, 3)
    for a, b in zip(got, (sc, ve)):
        if dtype == np.float64:
            assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b))
            continue
        ulp = np.spacing(np.maximum(np.abs(a), np.abs(b)))
        assert np.all(np.abs(a.astype(np.float64) - b) <= 8 * ulp.astype(np.float64) + 1e-30)
        assert np.mean(a != b) <= 0.01
    for r, o in zip(rows, o_rows):
        for k in ("energy", "gradient", "magnetic"):
            np.testing.assert_allclose(r[k], o[k], rtol=2e-5 if dtype == np.float32 else 1e-12)
