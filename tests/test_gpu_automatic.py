"""gft_set_kernel with kind 0 and nothing else asked for: a fresh handle's choice again (GPU).

Each lattice is on one side of the automatic rule with the tile and march gft_create chooses and on
the other with those of the call before: SM mixed 128^3 takes tiles in marches of 12 planes, not of
32; SM FP64 96 x 96 x 240 would take 4 x 16 tiles in marches of 8, not the 8 x 16 of its own.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,model,shape,before,name", [
    ("mixed", 1, (128, 128, 128), (2, 0, 32), "tiled_step_kernel"),
    ("mixed", 2, (192, 192, 192), (1, 0, 32), "tiled_step_kernel"),
    ("mixed", 1, (64, 64, 48), (2, 2, 1), "fast_step_kernel"),
    ("fp64", 1, (96, 96, 240), (2, 2, 8), "fast_step_kernel"),
    ("fp64", 1, (3, 384, 512), (2, 3, 32), "tiled_step_kernel"),
    ("fp64", 2, (3, 768, 512), (1, 0, 32), "tiled_step_kernel"),
])
def test_kind_0_restores_the_choice_made_at_creation(form, model, shape, before, name):
    from gftevolver_b200 import Evolver, InitialData, LatticeParams
    nx, ny, nz = shape
    p = LatticeParams(model=model, nx=nx, ny=ny, nz=nz, energy_every=2)
    ic = InitialData(seed=5, mean=[1.0 if model == 1 else 0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1, eps_sigma=0.1)
    out = []
    for restored in (False, True):
        with Evolver(p, form=form) as ev:
            if restored:
                ev.set_kernel(*before)
                ev.set_kernel()
            assert ev.step_kernel_name == name
            ev.init_fields(ic)
            rows = ev.evolve(3)
            out.append((rows, ev.launch_count, *ev.download()))
    (rows, launches, sc, ve), again = out
    assert rows == again[0] and launches == again[1]
    np.testing.assert_array_equal(sc, again[2])
    np.testing.assert_array_equal(ve, again[3])


def test_kind_0_keeps_a_tile_it_is_given():
    """Asked for a tile or march, kind 0 chooses between it and one thread per site, as before."""
    from gftevolver_b200 import Evolver, LatticeParams
    with Evolver(LatticeParams(model=1, nx=64, ny=64, nz=64), form="mixed") as ev:
        assert ev.step_kernel_name == "fast_step_kernel"
        ev.set_kernel(0, 2, 8)  # 4 x 16 tiles in marches of 8: 512 of them, under a wave
        assert ev.step_kernel_name == "fast_step_kernel"
        ev.set_kernel(0, 0, 2)  # 8 x 32 tiles in marches of 2: 512, 1.7 waves
        assert ev.step_kernel_name == "tiled_step_kernel"
        ev.set_kernel()
        assert ev.step_kernel_name == "fast_step_kernel"


@pytest.mark.parametrize("form,model,family", [("mixed", 1, 0), ("fp64", 1, 0), ("mixed", 2, 2), ("fp64", 2, 1)])
def test_kind_1_is_one_thread_per_site_on_small_lattices_too(form, model, family):
    """Kind 1 on 16,384 sites, which the automatic choice divides over warps, against the same fields
    twice along x, which are too many for that: the same kernel leaves the same bits, twice."""
    from gftevolver_b200 import Evolver, InitialData, LatticeParams
    ic = InitialData(seed=9, mean=[1.0 if model == 1 else 0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1, eps_sigma=0.1)
    make = lambda nx: Evolver(LatticeParams(model=model, nx=nx, ny=32, nz=32, higgs_family=family, energy_every=2),  # noqa: E731
                              form=form)
    with make(16) as small, make(32) as large:
        small.init_fields(ic)
        sc, ve = small.download()
        large.upload(*(np.concatenate([a, a], 1) for a in (sc, ve)), 0)
        small.set_kernel(1)
        small.evolve(3)
        large.evolve(3)
        assert large.step_kernel_name == small.step_kernel_name == "fast_step_kernel"
        for a, b in zip(small.download(), large.download()):
            np.testing.assert_array_equal(np.concatenate([a, a], 1), b)


@pytest.mark.parametrize("form,model,shape", [
    ("mixed", 1, (80, 80, 80)),     # 16 x 16 tiles fill 0.6 of a wave: 56 us a step, one thread per site 39
    ("mixed", 1, (96, 100, 96)),    # 4 x 32 tiles, one wave: 81 / 64
    ("mixed", 2, (200, 100, 144)),  # 4 x 16 tiles only: 275 / 240
    ("fp64", 1, (128, 132, 128)),   # 4 x 32 tiles only: 433 / 298
])
def test_lattices_that_tile_badly_run_one_thread_per_site(form, model, shape):
    from gftevolver_b200 import Evolver, LatticeParams
    nx, ny, nz = shape
    with Evolver(LatticeParams(model=model, nx=nx, ny=ny, nz=nz), form=form) as ev:
        assert ev.step_kernel_name == "fast_step_kernel"


@pytest.mark.parametrize("model", [1, 2])
def test_an_edge_of_16_takes_16_x_16_tiles(model):
    """z divides into 16 but not 32: 16 x 16 tiles, not 4 x 16, by the partial sums of the energy row,
    whose order is the tiles'."""
    from gftevolver_b200 import Evolver, InitialData, LatticeParams
    p = LatticeParams(model=model, nx=144, ny=144, nz=144, energy_every=1)
    ic = InitialData(seed=5, mean=[1.0 if model == 1 else 0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1, eps_sigma=0.1)
    rows = []
    for kernel in (None, (2, 3, 12), (2, 2, 12)):
        with Evolver(p, form="mixed") as ev:
            if kernel:
                ev.set_kernel(*kernel)
            assert ev.step_kernel_name == "tiled_step_kernel"
            ev.init_fields(ic)
            rows.append(ev.evolve(1))
    assert rows[0] == rows[1] != rows[2]


@pytest.mark.parametrize("form", ["mixed", "fp64"])
@pytest.mark.parametrize("shape,divided", [((16, 32, 32), True), ((17, 32, 32), False)])
def test_the_divided_step_serves_16384_sites_and_no_more(form, shape, divided):
    """Which step runs, by its bits: the divided one sums a site's forces in another order."""
    from gftevolver_b200 import Evolver, InitialData, LatticeParams
    ic = InitialData(seed=9, mean=[0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1, eps_sigma=0.1)
    out = []
    for kind in (0, 1):
        with Evolver(LatticeParams(model=2, nx=shape[0], ny=shape[1], nz=shape[2]), form=form) as ev:
            ev.set_kernel(kind)
            ev.init_fields(ic)
            ev.evolve(2)
            out.append(ev.download())
    same = all(np.array_equal(a, b) for a, b in zip(*out))
    assert same != divided
