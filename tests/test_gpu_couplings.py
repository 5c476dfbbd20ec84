"""Every term of the update at once, on every route of the throughput forms (GPU).

All couplings of the two-doublet potential (the CP-violating ones too), three different spacings,
damped first steps: against the FP64 oracle.  Bars after 4 steps: the FP64 form 1e-12 of the fields, the
mixed form 6e-6; sums of the potential, gradient and kinetic energy 1e-11 and 1e-5 relative.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CP = dict(l6r=0.03, l7r=-0.04, m12i=0.07, l4m5=0.05, l5i=-0.03, l6i=0.02, l7i=0.06)
SPACING = dict(dx=1.3, dy=0.9, dz=1.1, damping=0.3, nt_damped=2)


def _params(oracle_mod, model, shape, family=0, **kw):
    nx, ny, nz = shape
    extra = CP if model == 2 else {}
    return oracle_mod.Params(model=model, nx=nx, ny=ny, nz=nz, higgs_family=family, energy_every=3, gauss_every=3,
                             **SPACING, **extra, **kw)


def _fields(oracle_mod, op, dtype):
    ic = oracle_mod.ICSpec(seed=41, mean=[0.6, -0.3, 0.2, 0.7, 0.5, 0.4, -0.6, 0.3] if op.model == 2 else [0.5] * 8,
                           sigma=[0.2] * 8, theta_sigma=0.2, eps_sigma=0.2)
    sc, ve = oracle_mod.init_fields(op, ic, np.float64)
    rng = np.random.default_rng(8)
    dw = ve.shape[-1] // 3
    sc[0] -= 0.02 * rng.standard_normal(sc[0].shape)  # momenta of the doublets and the phases
    ve[0][..., ::dw] -= 0.02 * rng.standard_normal(ve[0][..., ::dw].shape)
    return sc.astype(dtype), ve.astype(dtype)


def _compare(oracle_mod, op, form, rows, got, sc, ve):
    sc, ve = sc.astype(np.float64), ve.astype(np.float64)
    o_rows, _ = oracle_mod.evolve(op, sc, ve, 4)
    for a, b in zip(got, (sc, ve)):
        err = np.max(np.abs(a.astype(np.float64) - b))
        assert err <= (1e-12 * np.max(np.abs(b)) if form == "fp64" else 6e-6)
    assert [r["time_iter"] for r in rows] == [0, 3]
    for r, o in zip(rows, o_rows):
        for k in ("potential", "gradient", "kinetic"):
            assert abs(r[k] - o[k]) <= (1e-11 if form == "fp64" else 1e-5) * abs(o[k]), k


@pytest.mark.parametrize("form,model,family,shape,kernel,name", [
    ("mixed", 1, 0, (12, 20, 24), None, "fast"), ("fp64", 1, 0, (12, 20, 24), None, "fast"),
    ("mixed", 2, 0, (12, 20, 24), None, "fast"), ("fp64", 2, 0, (12, 20, 24), None, "fast"),
    ("mixed", 2, 1, (12, 20, 24), None, "fast"), ("fp64", 2, 2, (12, 20, 24), None, "fast"),
    ("mixed", 1, 0, (11, 40, 64), None, "fast"), ("fp64", 1, 0, (11, 40, 50), None, "fast"),
    ("mixed", 2, 0, (11, 40, 50), None, "fast"), ("fp64", 2, 0, (11, 40, 64), None, "fast"),
    ("mixed", 2, 2, (11, 40, 50), None, "fast"), ("fp64", 2, 1, (11, 40, 64), None, "fast"),
    ("mixed", 1, 0, (7, 48, 96), (2, 0, 3), "tiled"), ("mixed", 1, 0, (7, 48, 96), (2, 2, 3), "tiled"),
    ("mixed", 1, 0, (7, 48, 96), (2, 3, 3), "tiled"), ("mixed", 2, 0, (7, 48, 96), (2, 0, 3), "tiled"),
    ("mixed", 2, 0, (7, 48, 96), (2, 1, 3), "tiled"), ("fp64", 1, 0, (7, 48, 96), (2, 0, 3), "tiled"),
    ("fp64", 1, 0, (7, 48, 96), (2, 1, 3), "tiled"), ("fp64", 1, 0, (2, 416, 384), None, "tiled"),
    ("fp64", 2, 0, (2, 320, 304), None, "tiled"),
])
def test_all_couplings_spacings_and_damping(oracle_mod, form, model, family, shape, kernel, name):
    from gftevolver_b200 import Evolver, LatticeParams
    op = _params(oracle_mod, model, shape, family)
    sc, ve = _fields(oracle_mod, op, np.float64 if form == "fp64" else np.float32)
    with Evolver(LatticeParams(**op.__dict__), form=form) as ev:
        if kernel:
            ev.set_kernel(*kernel)
        assert ev.step_kernel_name == name + "_step_kernel"
        ev.upload(sc, ve, 0)
        rows = ev.evolve(4)
        assert ev.last_warnings == 0
        got = ev.download()
    _compare(oracle_mod, op, form, rows, got, sc, ve)


@pytest.mark.parametrize("model", [1, 2])
def test_ensemble_of_all_couplings_spacings_and_damping(oracle_mod, model):
    from gftevolver_b200 import Ensemble, LatticeParams
    ops = [_params(oracle_mod, model, (7, 48, 96)), _params(oracle_mod, model, (10, 32, 32), g=0.6)]
    fields = [_fields(oracle_mod, op, np.float32) for op in ops]
    with Ensemble([LatticeParams(**op.__dict__) for op in ops]) as ens:
        for m, (sc, ve) in enumerate(fields):
            ens.upload(m, sc, ve, 0)
        rows = ens.evolve(4)
        got = [ens.download(m) for m in range(2)]
    for m, op in enumerate(ops):
        _compare(oracle_mod, op, "mixed", rows[m], got[m], *fields[m])
