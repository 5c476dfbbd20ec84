"""The x-march's carried loops at the ends of marches (GPU).

A tile's site reads nothing of the plane x - 1: the lower loops of that plane
come from the site before it in the march, or, at the start of a march, from the
values of the plane before it (site_carry).  The cases are the shortest lattices
and marches (every site starts a march, marches of one and two planes left over,
rings with fewer planes than buffers), with and without Fixed x faces, whose
frozen sites hand their loops on unevolved.  Bars: the FP64 form 1e-12 relative
to the FP64 oracle after 6 steps, the mixed form 6e-6 absolute.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fixed", [0, 1], ids=["periodic", "fixed_x"])
@pytest.mark.parametrize("form,model", [("fp64", 1), ("mixed", 1), ("mixed", 2)])
@pytest.mark.parametrize("nx,march", [(1, 1), (2, 1), (2, 8), (3, 2), (4, 3), (5, 4), (7, 3)])
def test_march_ends_match_oracle(oracle_mod, form, model, nx, march, fixed):
    from gftevolver_b200 import Evolver, LatticeParams
    op = oracle_mod.Params(model=model, nx=nx, ny=24, nz=96, energy_every=3, fixed_axes=fixed)
    ic = oracle_mod.ICSpec(seed=17, mean=[1.0 if model == 1 else 0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1,
                           eps_sigma=0.1)
    sc, ve = oracle_mod.init_fields(op, ic, np.float64)
    with Evolver(LatticeParams(**op.__dict__), form=form) as ev:
        ev.set_kernel(2, 0, march)
        assert ev.step_kernel_name == "tiled_step_kernel"
        ev.upload(sc, ve, 0)
        ev.evolve(6)
        assert ev.last_warnings == 0
        g_sc, g_ve = ev.download()
    oracle_mod.evolve(op, sc, ve, 6)
    for a, b in ((g_sc, sc), (g_ve, ve)):
        err = np.max(np.abs(a.astype(np.float64) - b))
        assert err <= (1e-12 * np.max(np.abs(b)) if form == "fp64" else 6e-6)


@pytest.mark.parametrize("fixed", [0, 7], ids=["periodic", "fixed"])
def test_fp64_default_tile_matches_one_thread_per_site(fixed):
    """The FP64 step's own 8 x 16 tile, which only the automatic choice takes, on a lattice thin in x
    with enough tiles for it, against the oracle-pinned one-thread-per-site step: every loop and
    transport that sites hand over within a tile, across its halo row and column and over the wrap.
    Bar: 1e-12 of the fields after 5 steps, the rows within 1e-12 of the total energy."""
    from gftevolver_b200 import Evolver, InitialData, LatticeParams
    p = LatticeParams(model=1, nx=3, ny=384, nz=512, energy_every=2, gauss_every=2, fixed_axes=fixed)
    ic = InitialData(seed=5, mean=[1.0] * 8, sigma=[0.1] * 8, theta_sigma=0.1, eps_sigma=0.1)
    out = []
    for kind in (0, 1):
        with Evolver(p, form="fp64") as ev:
            if kind:
                ev.set_kernel(kind, 0, 32)
            assert ev.step_kernel_name == ("fast_step_kernel" if kind else "tiled_step_kernel")
            ev.init_fields(ic)
            rows = ev.evolve(5)
            out.append((*ev.download(), rows))
    for a, b in zip(out[0][:2], out[1][:2]):
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
    for a, b in zip(out[0][2], out[1][2]):
        for k in ("energy", "potential", "gradient", "kinetic", "magnetic", "electric"):
            assert abs(a[k] - b[k]) <= 1e-12 * abs(b["energy"]), k


@pytest.mark.parametrize("fixed", [0, 7], ids=["periodic", "fixed"])
@pytest.mark.parametrize("nx", [1, 2, 5, 34])
def test_fp64_two_doublets_tile_matches_one_thread_per_site(nx, fixed):
    """The FP64 2HDM's 8 x 16 tile over its ring of two planes, against the oracle-pinned
    one-thread-per-site step: marches shorter than the ring, odd ones, and a second march of two
    planes.  Bars as above."""
    from gftevolver_b200 import Evolver, InitialData, LatticeParams
    ny, nz = (768, 512) if nx < 34 else (384, 512)
    p = LatticeParams(model=2, nx=nx, ny=ny, nz=nz, energy_every=2, gauss_every=2, fixed_axes=fixed)
    ic = InitialData(seed=5, mean=[0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1, eps_sigma=0.1)
    out = []
    for kind in (0, 1):
        with Evolver(p, form="fp64") as ev:
            if kind:
                ev.set_kernel(kind, 0, 32)
            assert ev.step_kernel_name == ("fast_step_kernel" if kind else "tiled_step_kernel")
            ev.init_fields(ic)
            rows = ev.evolve(5)
            out.append((*ev.download(), rows))
    for a, b in zip(out[0][:2], out[1][:2]):
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
    for a, b in zip(out[0][2], out[1][2]):
        for k in ("energy", "potential", "gradient", "kinetic", "magnetic", "electric"):
            assert abs(a[k] - b[k]) <= 1e-12 * abs(b["energy"]), k


def test_one_plane_of_small_tiles_keeps_every_partial_row():
    """A lattice one plane thick whose edges admit 4 x 16 tiles only: 1,203 of them, more than the
    one-thread-per-site step has blocks, each with its row of partial energies.  The rows of the two
    steps agree as their sums do: 1e-5 of the total energy, the mixed form's bar."""
    from gftevolver_b200 import Evolver, InitialData, LatticeParams
    p = LatticeParams(model=1, nx=1, ny=1604, nz=48, energy_every=1)
    ic = InitialData(seed=5, mean=[1.0] * 8, sigma=[0.1] * 8, theta_sigma=0.1, eps_sigma=0.1)
    out = []
    for kind in (0, 1):
        with Evolver(p, form="mixed") as ev:
            if kind:
                ev.set_kernel(kind, 0, 32)
            assert ev.step_kernel_name == ("fast_step_kernel" if kind else "tiled_step_kernel")
            ev.init_fields(ic)
            out.append(ev.evolve(3))
    for a, b in zip(*out):
        for k in ("energy", "potential", "gradient", "kinetic", "magnetic", "electric"):
            assert abs(a[k] - b[k]) <= 1e-5 * abs(b["energy"]), k


@pytest.mark.parametrize("model,shape,kind", [(1, (16, 16, 16), 0), (1, (40, 40, 40), 0), (1, (8, 24, 96), 2),
                                              (2, (16, 16, 16), 0), (2, (40, 40, 40), 0)])
def test_fp64_step_renormalises_links_of_float_words(oracle_mod, model, shape, kind):
    """FP64 form, links of float words (unit to 6e-8): the step leaves them unit to double rounding,
    as the reference's renormalisation does.  Bar: |U|^2 - 1 of a link whose four words are each
    rounded thrice, 8 ulp of 2.2e-16 with the norm's own evaluation."""
    from gftevolver_b200 import Evolver, LatticeParams
    op = oracle_mod.Params(model=model, nx=shape[0], ny=shape[1], nz=shape[2])
    ic = oracle_mod.ICSpec(seed=23, mean=[1.0 if model == 1 else 0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1,
                           eps_sigma=0.1)
    sc, ve = (a.astype(np.float64) for a in oracle_mod.init_fields(op, ic, np.float32))
    with Evolver(LatticeParams(**op.__dict__), form="fp64") as ev:
        if kind:
            ev.set_kernel(kind, 0, 4)
        ev.upload(sc, ve, 0)
        ev.evolve(1)
        new = ev.download()[1][0].reshape(*shape, 3, 5)[..., 1:]  # the step from iteration 0 writes slot 0
    assert np.max(np.abs(np.sum(new * new, -1) - 1.0)) <= 8 * 2.0 ** -52
