"""Reference-layout fields into the level arrays and back (GPU): the staged runs of a
block of 128 sites at their edges (one site, a block less one, a block, a block and
one, several), every record shape, both storages and host types, and device buffers
aligned to a single element.  Quaternion records come back as they went in, to the
storage's rounding; generator records of the throughput forms to 8 roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["mixed", "fp64", "ref32", "ref64"])
@pytest.mark.parametrize("host", ["f32", "f64"])
@pytest.mark.parametrize("model,family,gen", [(1, 0, 0), (2, 0, 0), (2, 1, 0), (2, 2, 0), (1, 0, 1), (2, 1, 1), (2, 2, 1)])
def test_round_trip(form, host, model, family, gen):
    import torch

    from gftevolver_b200 import Evolver, LatticeParams
    dtype = torch.float64 if host == "f64" else torch.float32
    for shape in ((1, 1, 1), (1, 127, 1), (2, 8, 8), (3, 43, 1), (5, 9, 31)):
        p = LatticeParams(model=model, nx=shape[0], ny=shape[1], nz=shape[2], higgs_family=family, generator_rep=gen)
        nsc, nve = 2 * p.nsite * p.nsc, 2 * p.nsite * p.nve
        g = torch.Generator(device="cuda").manual_seed(7)
        # buffers one element off the allocation's alignment; rotations small enough to invert
        src = [0.1 * torch.randn(n + 1, generator=g, device="cuda", dtype=dtype).clamp(-3, 3)[1:] for n in (nsc, nve)]
        out = [torch.full((n + 1,), float("nan"), device="cuda", dtype=dtype)[1:] for n in (nsc, nve)]
        torch.cuda.synchronize()
        with Evolver(p, form=form) as ev:
            ev.upload_device(src[0].data_ptr(), src[1].data_ptr(), host == "f64", 0)
            ev.download_device(out[0].data_ptr(), out[1].data_ptr(), host == "f64")
            sc, ve = ev.download(np.float64 if host == "f64" else np.float32)
        single = host == "f32" or form in ("mixed", "ref32")
        for k, (a, b) in enumerate(zip(src, out)):
            want = a.float().to(dtype) if single else a
            if gen and k == 1 and form in ("mixed", "fp64"):
                # w -> (cos|w|, sin|w| w/|w|) -> w, |w| <= 0.3 sqrt(3) = 0.52: the words are rounded once on
                # storing (relative 2^-24 or 2^-53); inverting multiplies that by tan|w|/|w| < 1.2, and the
                # functions and the final rounding add a few units more
                eps = 2.0 ** -24 if single else 2.0 ** -53
                assert (b.double() - a.double()).abs().max().item() <= 8 * 0.52 * eps
            else:
                assert torch.equal(b, want), (shape, k)
        assert np.array_equal(sc.ravel(), out[0].cpu().numpy()) and np.array_equal(ve.ravel(), out[1].cpu().numpy())
