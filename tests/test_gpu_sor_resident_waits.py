"""The chip-resident SOR's bounded waits: a wait that runs out is reported, and
the context steps again as a new one after the next upload."""
import ctypes as C

import numpy as np
import pytest

import oracle
from les_halo_b200 import GpuLes, abi, fields as FL, synthetic_case
from tests.helpers import assert_bitexact

pytestmark = pytest.mark.gpu


def _case(dims, seed):
    return synthetic_case(*dims, seed=seed, dx=4.0, dy=4.0, masks_and_poisson=oracle.masks_and_poisson)


def _void(g, nsteps=1):
    """Steps whose waits run out (one poll, where a word takes a trip through L2)."""
    abi.check(abi.lib().les_ctx_set_sor_wait(g.ctx, 1))
    g.warmup(1)
    g.step(1, nsteps)


def _times_out(call, *a):
    with pytest.raises(abi.LesError) as e:
        call(*a)
    assert e.value.status == abi.LES_ERR_TIMEOUT


@pytest.mark.parametrize("dims", [(61, 47, 35), (150, 150, 90)])
@pytest.mark.parametrize("nsteps", [1, 3])
@pytest.mark.parametrize("at_upload", [False, True])
def test_a_void_step_leaves_nothing_behind(require_gpu, dims, nsteps, at_upload):
    # the abandoned launch's words carry the tags of the next one's first
    # half-sweeps: with another state uploaded they must not be taken for its own
    a, b = _case(dims, 5), _case(dims, 9)
    hb = b.host_fields()
    g = GpuLes(a.copy())
    _void(g, nsteps)
    if at_upload:
        _times_out(abi.check, abi.lib().les_ctx_upload(g.ctx, C.byref(hb)))
    else:
        _times_out(g.sync)
    g.sync()  # reported once
    abi.check(abi.lib().les_ctx_set_sor_wait(g.ctx, 0))
    abi.check(abi.lib().les_ctx_upload(g.ctx, C.byref(hb)))
    g.warmup(1)
    g.step(1, 2)
    got, m = g.download(FL.STATE), g.metrics()
    g.close()
    ref = GpuLes(b.copy())
    abi.check(abi.lib().les_ctx_set_sor_path(ref.ctx, 1))
    ref.warmup(1)
    ref.step(1, 2)
    assert_bitexact(got, ref.download(FL.STATE), *dims, FL.STATE)
    assert m["sor_iters"] == ref.metrics()["sor_iters"]
    ref.close()
