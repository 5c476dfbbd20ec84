"""The ring of two planes when a wait gives up (GPU): the FP64 2HDM's tiles.

As test_gpu_waits.py, for the ring whose copy lands during a site's second half: it is waited for ahead of
the next plane, by a vote of each warp, with a barrier more where the tile wraps.  A limit of 1 ns fails
at once; limits of about a copy's latency let some waits pass, so that others give up in the middle of a
march: either outcome is right, and the handle is usable after it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_plane_ring_gives_up_and_the_handle_recovers():
    from gftevolver_b200 import Evolver, GftError, InitialData, LatticeParams
    from gftevolver_b200 import _lib
    p = LatticeParams(model=2, nx=40, ny=320, nz=304, energy_every=2, gauss_every=2)
    ic = InitialData(seed=5, mean=[0.7] * 8, sigma=[0.1] * 8, theta_sigma=0.1, eps_sigma=0.1)
    with Evolver(p, form="fp64") as ev:
        assert ev.step_kernel_name == "tiled_step_kernel"
        ev.init_fields(ic)
        rows = ev.evolve(3)
        want = ev.download()
    with Evolver(p, form="fp64") as ev:
        for limit in (1, 1200, 1600, 2000, 3000, 5000):
            ev.set_wait_limit(limit)
            ev.init_fields(ic)
            try:
                ev.evolve(1)
                assert limit > 1
            except GftError as err:
                assert err.code == _lib.GFT_E_TIMEOUT
        ev.set_wait_limit(0)
        ev.init_fields(ic)
        assert ev.evolve(3) == rows and ev.last_warnings == 0
        for a, b in zip(ev.download(), want):
            np.testing.assert_array_equal(a, b)
