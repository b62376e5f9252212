"""The chip-resident SOR (one launch per step) against the per-colour sweeps,
bit for bit: state, iteration count, residual."""
import numpy as np
import pytest

import oracle
from les_halo_b200 import GpuLes, abi, fields as FL, synthetic_case
from tests.helpers import assert_bitexact

pytestmark = pytest.mark.gpu

KEYS = ("sor_iters", "sor", "rhsav", "pav", "p_centre")


def _pair(dims, seed=5, pjuge=None, nmaxp=50, steps=2, dx=4.0):
    case = synthetic_case(*dims, seed=seed, nmaxp=nmaxp, dx=dx, dy=dx, masks_and_poisson=oracle.masks_and_poisson)
    if pjuge is not None:
        case.params.pjuge = pjuge
    got = []
    for per_colour in (0, 1):
        g = GpuLes(case.copy())
        abi.check(abi.lib().les_ctx_set_sor_path(g.ctx, per_colour))
        g.warmup(1)
        g.step(1, steps - 1)
        n0 = g.launches()
        g.step(steps, 1)
        n = g.launches() - n0
        got.append((g.download(FL.STATE), g.metrics(), n))
        g.close()
    (a, ma, la), (b, mb, _) = got
    assert la < 24, "the passes ran"  # a step of passes launches 50 more
    assert_bitexact(a, b, *dims, FL.STATE)
    for k in KEYS:
        assert np.float32(ma[k]).view(np.uint32) == np.float32(mb[k]).view(np.uint32), k
    return mb


# one CTA (even and odd jm), many; tiles of two columns, clipped last tiles;
# one segment per column to five, planes that fill it and that do not; odd
# extents; segments of 8 to 64 planes, the rhs in shared and in global memory
@pytest.mark.parametrize("dims", [(24, 20, 16), (9, 9, 5), (24, 9, 12), (16, 8, 3), (40, 33, 14), (61, 47, 35),
                                  (64, 48, 33), (30, 70, 64), (150, 150, 90), (257, 203, 61), (180, 180, 80),
                                  (300, 200, 40), (96, 250, 79)])
def test_resident_equals_per_colour(require_gpu, dims):
    m = _pair(dims)
    assert m["sor_iters"] == 50


@pytest.mark.parametrize("nmaxp", [1, 2, 7])
@pytest.mark.parametrize("dims", [(24, 20, 16), (61, 47, 35)])
def test_resident_iteration_caps(require_gpu, dims, nmaxp):
    assert _pair(dims, nmaxp=nmaxp)["sor_iters"] == nmaxp


@pytest.mark.parametrize("dims", [(24, 20, 16), (61, 47, 35), (130, 101, 50)])
@pytest.mark.parametrize("stop", [1, 6, 19, 20])
def test_resident_stops_where_the_exact_residual_says(require_gpu, dims, stop):
    # the residual after `stop` iterations as the threshold: not met there
    # (undecidable by the FP32 bound, summed again exactly), and met with the
    # next larger float
    r = np.float32(_pair(dims, nmaxp=stop, pjuge=-1.0, steps=1)["sor"])
    above = float(np.nextafter(r, np.float32(np.inf)))
    assert _pair(dims, nmaxp=20, pjuge=above, steps=1)["sor_iters"] == stop
    assert _pair(dims, nmaxp=20, pjuge=float(r), steps=1)["sor_iters"] == min(stop + 1, 20)


def test_resident_contexts_side_by_side(require_gpu):
    # several contexts' launches queued on their own streams together
    cases = [synthetic_case(*d, seed=s, masks_and_poisson=oracle.masks_and_poisson)
             for s, d in enumerate([(61, 47, 35), (150, 150, 90), (96, 80, 40), (130, 101, 50)])]
    alone, together = [], []
    for c in cases:
        g = GpuLes(c.copy())
        g.warmup(1)
        g.step(1, 6)
        alone.append(g.download(FL.STATE))
        g.close()
    gs = [GpuLes(c.copy()) for c in cases]
    for g in gs:
        g.warmup(1)
    for n in range(1, 7):
        for g in gs:
            g.step(n, 1)
    for c, g, a in zip(cases, gs, alone):
        g.sync()
        assert_bitexact(g.download(FL.STATE), a, c.ip, c.jp, c.kp, FL.STATE)
    for g in gs:
        g.close()
