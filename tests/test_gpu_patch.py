"""The one-thread-per-site kernels' block shapes and the divided step of small lattices (GPU).

Edges along z that leave a block of 32 x 4 threads idle take other patches; lattices up to 16,384
sites divide a site's update over warps.  The sizes lie on both sides of that line and at the
patches' remainders (a row of 33 sites, rows narrower than a patch, one site).  Bars: the FP64 form
1e-12 of the FP64 oracle after 4 steps, the mixed form 6e-6; the Gauss pass against the oracle's on
the same fields to FP64 rounding.
(Energies: test_gpu_parity.py, whose lattices are small; the oracle's 1 - cos of a small
angle is itself off by 1e-16 x 4 / dt^2 g'^2 = 1e-12 a site here.)
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("model,family,fixed", [(1, 0, 0), (1, 0, 5), (2, 0, 0), (2, 1, 2), (2, 2, 4)])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 5, 7), (2, 3, 33), (16, 32, 32), (29, 17, 34), (7, 33, 75),
                                   (5, 65, 64), (3, 200, 29), (2, 100, 101)])
def test_any_shape_matches_oracle(oracle_mod, form, model, family, fixed, shape):
    from gftevolver_b200 import Evolver, LatticeParams
    if fixed and min(shape) < 3:
        pytest.skip("a Fixed axis needs inner sites")
    nx, ny, nz = shape
    op = oracle_mod.Params(model=model, nx=nx, ny=ny, nz=nz, higgs_family=family, fixed_axes=fixed, energy_every=2,
                           gauss_every=3)
    ic = oracle_mod.ICSpec(seed=9, mean=[1.0 if model == 1 else 0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1,
                           eps_sigma=0.1)
    sc, ve = oracle_mod.init_fields(op, ic, np.float64)
    dw = op.nve // 3  # momenta on the hypercharge phases: a Gauss residual to compare
    ve[0][..., ::dw] += 1e-3 * np.random.default_rng(3).standard_normal(ve[0][..., ::dw].shape)
    with Evolver(LatticeParams(**op.__dict__), form=form) as ev:
        assert ev.step_kernel_name == "fast_step_kernel"
        ev.upload(sc, ve, 0)
        rows = ev.evolve(4)
        g_sc, g_ve = ev.download()
    if form == "mixed":  # the oracle from the words the evolver holds
        sc, ve = sc.astype(np.float32).astype(np.float64), ve.astype(np.float32).astype(np.float64)
    o_rows, _ = oracle_mod.evolve(op, sc, ve, 4)
    fp64 = form == "fp64"
    for a, b in ((g_sc, sc), (g_ve, ve)):
        err = np.max(np.abs(a.astype(np.float64) - b))
        assert err <= (1e-12 * np.max(np.abs(b)) if fp64 else 6e-6)
    assert [r["time_iter"] for r in rows] == [r["time_iter"] for r in o_rows]
    # the Gauss pass of step 3 against the oracle's on the very fields it saw: both in FP64 from the same
    # words, a dozen terms of order one at most per site and constraint
    gi, gm, _ = oracle_mod.gauss(op, g_sc.astype(np.float64), g_ve.astype(np.float64), 3)
    assert rows[-1]["time_iter"] == 3 and rows[-1]["has_gauss"]
    np.testing.assert_allclose(rows[-1]["gauss_max"], gm, rtol=1e-11, atol=2e-15)
    np.testing.assert_allclose(rows[-1]["gauss_int"], gi, rtol=1e-11, atol=2e-15 * nx * ny * nz)
