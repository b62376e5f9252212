"""The chip-resident SOR with segments of 40 planes and more, whose bounds are
summed once per batch of iterations: stops in and around the batches, against
the per-colour sweeps."""
import numpy as np
import pytest

import oracle
from les_halo_b200 import GpuLes, abi, fields as FL, synthetic_case
from tests.helpers import assert_bitexact

pytestmark = pytest.mark.gpu


def _run(dims, nmaxp, pjuge, per_colour=0):
    case = synthetic_case(*dims, seed=5, nmaxp=nmaxp, dx=4.0, dy=4.0, masks_and_poisson=oracle.masks_and_poisson)
    case.params.pjuge = pjuge
    g = GpuLes(case)
    abi.check(abi.lib().les_ctx_set_sor_path(g.ctx, per_colour))
    g.warmup(1)
    g.step(1, 1)
    assert abi.lib().les_ctx_sor_resident(g.ctx) == 1 - per_colour
    out = g.download(FL.STATE), g.metrics()
    g.close()
    return out


# segments of 40, 48 and 64 planes, one CTA and many
@pytest.mark.parametrize("dims", [(8, 9, 40), (10, 8, 45), (8, 8, 60), (180, 180, 80), (150, 150, 90), (257, 203, 61)])
def test_stops_in_long_segments(require_gpu, dims):
    for stop, cap in [(1, 2), (3, 50), (4, 5), (5, 50), (8, 9), (11, 14), (13, 14), (14, 14)]:
        r = np.float32(_run(dims, stop, -1.0)[1]["sor"])
        pj = float(np.nextafter(r, np.float32(np.inf)))
        (a, ma), (b, mb) = _run(dims, cap, pj), _run(dims, cap, pj, per_colour=1)
        assert ma["sor_iters"] == mb["sor_iters"] == stop, (stop, cap)
        for k in ("sor", "rhsav", "pav", "p_centre"):
            assert np.float32(ma[k]).view(np.uint32) == np.float32(mb[k]).view(np.uint32), (stop, cap, k)
        assert_bitexact(a, b, *dims, FL.STATE)
