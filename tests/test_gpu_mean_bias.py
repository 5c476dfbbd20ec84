"""The mixed form's doublets do not drift as a whole (GPU).

The Laplacian of a constant is zero and a float word rounds to nearest, so the mean deviation of the
mixed form's doublets from the FP64 form's stays far below that of a word.  Bar after t = 1:
  * rounding: each step rounds a word by 2^-24 / sqrt(12) rms at most (|phi| < 2), a leapfrog adds n - j
    times the j-th rounding, and the Laplacian conserves the sum over sites: the mean of M words is off
    by 2^-24 / sqrt(12) sqrt(n^3 / 3 / M) rms, of which six;
  * the coefficients' rounding, 2^-24 relative: a mean force of up to one half (d/dphi of the potentials
    here) displaces by t^2 / 2 times that, twice for the weight and the coupling: 2^-25.
Every route of the step: divided over warps, one thread per site, tiles, an ensemble.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(oracle_mod, model, dt, spacing, shape):
    dx, dy, dz = spacing
    op = oracle_mod.Params(model=model, nx=shape[0], ny=shape[1], nz=shape[2], dt=dt, dx=dx, dy=dy, dz=dz, m1=0.37,
                           m2=0.41)
    ic = oracle_mod.ICSpec(seed=31, mean=[1.0 if model == 1 else 0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1,
                           eps_sigma=0.1)
    return op, ic


def _check(sc, exact, n):
    err = sc.astype(np.float64) - exact
    bar = 6 * 2.0 ** -24 / np.sqrt(12) * np.sqrt(n ** 3 / 3 / err[0].size) + 2.0 ** -25
    for level in err:
        assert abs(np.mean(level)) <= bar, (np.mean(level), bar)


@pytest.mark.parametrize("shape,kind", [((16, 32, 32), 0), ((40, 40, 40), 0), ((24, 32, 64), 2)],
                         ids=["divided", "one_thread_per_site", "tiles"])
@pytest.mark.parametrize("dt,spacing", [(0.05, (1.0, 1.0, 1.0)), (0.08, (1.0, 1.0, 1.0)), (0.06, (1.1, 0.9, 1.3))])
@pytest.mark.parametrize("model", [1, 2])
def test_mixed_doublets_keep_their_mean(oracle_mod, model, dt, spacing, shape, kind):
    from gftevolver_b200 import Evolver, LatticeParams
    op, ic = _case(oracle_mod, model, dt, spacing, shape)
    p = LatticeParams(**op.__dict__)
    sc, ve = oracle_mod.init_fields(op, ic, np.float32)
    n, out = round(1 / dt), []
    for form, dtype in (("mixed", np.float32), ("fp64", np.float64)):
        with Evolver(p, form=form) as ev:
            if kind and form == "mixed":
                ev.set_kernel(kind, 0, 8)
            ev.upload(sc.astype(dtype), ve.astype(dtype), 0)
            ev.evolve(n)
            out.append(ev.download()[0])
    _check(*out, n)


@pytest.mark.parametrize("model", [1, 2])
def test_ensemble_doublets_keep_their_mean(oracle_mod, model):
    from gftevolver_b200 import Ensemble, Evolver, LatticeParams
    cases = [_case(oracle_mod, model, dt, (1.0, 1.0, 1.0), (24, 32, 64)) for dt in (0.05, 0.08)]
    ps = [LatticeParams(**op.__dict__) for op, _ in cases]
    sc, ve = oracle_mod.init_fields(*cases[0], np.float32)
    n = 12
    with Ensemble(ps) as ens:
        for m in range(2):
            ens.upload(m, sc, ve, 0)
        ens.evolve(n)
        got = [ens.download(m)[0] for m in range(2)]
    for p, g in zip(ps, got):
        with Evolver(p, form="fp64") as ev:
            ev.upload(sc.astype(np.float64), ve.astype(np.float64), 0)
            ev.evolve(n)
            _check(g, ev.download()[0], n)
