"""The chip-resident SOR where it stops before its cap: what a stop costs, and
iteration count, residual and state around the batches its bounds travel in."""
import ctypes as C

import numpy as np
import pytest

import oracle
from les_halo_b200 import GpuLes, abi, fields as FL, synthetic_case
from tests.helpers import assert_bitexact

pytestmark = pytest.mark.gpu


def _case(dims, nmaxp, pjuge):
    case = synthetic_case(*dims, seed=5, nmaxp=nmaxp, dx=4.0, dy=4.0, masks_and_poisson=oracle.masks_and_poisson)
    case.params.pjuge = pjuge
    return case


def _run(dims, nmaxp, pjuge, per_colour=0):
    g = GpuLes(_case(dims, nmaxp, pjuge))
    abi.check(abi.lib().les_ctx_set_sor_path(g.ctx, per_colour))
    g.warmup(1)
    g.step(1, 1)
    out = g.download(FL.STATE), g.metrics()
    g.close()
    return out


def _stop_after(dims, m):
    """A threshold that the residual after m iterations is the first below."""
    r = np.float32(_run(dims, m, -1.0)[1]["sor"])
    return float(np.nextafter(r, np.float32(np.inf)))


def _sor_ms(dims, nmaxp, pjuge):
    """SOR time of one step from the same state, the least of three."""
    g = GpuLes(_case(dims, nmaxp, pjuge))
    L, ms, best = abi.lib(), (C.c_float * 9)(), []
    abi.check(L.les_ctx_set_timing(g.ctx, 4))
    for q in range(4):
        abi.check(L.les_ctx_upload(g.ctx, C.byref(g._hf)))
        g.warmup(1)
        g.step(1, 1)
        abi.check(L.les_ctx_phase_times(g.ctx, q, ms, 9))
        best.append(ms[5] + ms[6])
    its = g.metrics()["sor_iters"]
    g.close()
    return min(best[1:]), its


@pytest.mark.parametrize("dims", [(24, 20, 16), (61, 47, 35), (150, 150, 90)])
def test_a_stop_does_not_pay_for_the_cap(require_gpu, dims):
    # five iterations of 50 or of 2000: the same work.  (Looked at only after
    # the last iteration, the bounds cost 40 times as much with the second cap.)
    pj = _stop_after(dims, 5)
    t50, i50 = _sor_ms(dims, 50, pj)
    t2000, i2000 = _sor_ms(dims, 2000, pj)
    assert i50 == i2000 == 5
    assert t2000 < 2 * t50, (t50, t2000)


# one CTA and many; the single first batches, the ends and beginnings of the
# batches of four, and the last iterations before the cap
@pytest.mark.parametrize("dims", [(24, 20, 16), (24, 9, 12), (61, 47, 35), (30, 70, 64)])
@pytest.mark.parametrize("stop,cap", [(2, 50), (3, 50), (4, 50), (5, 50), (7, 50), (8, 50), (9, 50), (11, 14), (12, 14),
                                      (13, 14), (3, 4), (1, 2), (1, 3)])
def test_stops_around_the_batches(require_gpu, dims, stop, cap):
    pj = _stop_after(dims, stop)
    (a, ma), (b, mb) = _run(dims, cap, pj), _run(dims, cap, pj, per_colour=1)
    assert ma["sor_iters"] == mb["sor_iters"] == stop
    for k in ("sor", "rhsav", "pav", "p_centre"):
        assert np.float32(ma[k]).view(np.uint32) == np.float32(mb[k]).view(np.uint32), k
    assert_bitexact(a, b, *dims, FL.STATE)
