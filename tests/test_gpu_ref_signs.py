"""Signs of zero in the reference-arithmetic form (GPU).

The reference divides the components of a link's product by their norm, and a division keeps the
sign of a zero.  Links that hold zeros of either sign, in a vacuum where nothing else moves, pass
through every product of a step; the words come back as the oracle's, bit for bit.
"""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family", [None, 0, 2], ids=["sm", "2hdm", "2hdm_su2"])
@pytest.mark.parametrize("form,dtype", [("ref32", np.float32), ("ref64", np.float64)])
def test_normalised_products_keep_the_sign_of_zero(oracle_mod, form, dtype, family):
    from gftevolver_b200 import Evolver, LatticeParams
    model = 1 if family is None else 2
    shape = (4, 4, 4)
    op = oracle_mod.Params(model=model, nx=shape[0], ny=shape[1], nz=shape[2], higgs_family=family or 0)
    sc, ve = oracle_mod.init_fields(op, oracle_mod.ICSpec(seed=1, sigma=[0.0] * 8), dtype)
    words = np.array(list(itertools.product((-1.0, 1.0), *[(-0.0, 0.0)] * 3)), dtype)  # 16 links
    dw = ve.shape[-1] // 3
    for d in range(3):
        for at in ([1, 5] if family == 2 else [1]):
            # one link everywhere but for its zeros' signs, which differ from site to site
            sign = -1.0 if (d + at) % 2 else 1.0
            pick = [w for w in words if w[0] == sign]
            for n, s in enumerate(np.ndindex(*shape)):
                ve[:, s[0], s[1], s[2], dw * d + at:dw * d + at + 4] = pick[(n + d) % len(pick)]
    with Evolver(LatticeParams(**op.__dict__), form=form) as ev:
        ev.upload(sc, ve, 0)
        ev.evolve(1)
        g_sc, g_ve = ev.download()
    oracle_mod.evolve(op, sc, ve, 1)
    new = ve[0]
    assert np.any((new == 0) & np.signbit(new)), "the oracle keeps some zero negative"
    for a, b in ((g_sc, sc), (g_ve, ve)):
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(np.signbit(a), np.signbit(b))
