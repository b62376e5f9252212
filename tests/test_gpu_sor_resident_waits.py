"""The chip-resident SOR's bounded waits: a wait that runs out is reported, and
the context steps again as a new one after the next upload."""
import ctypes as C

import numpy as np
import pytest

import oracle
from les_halo_b200 import Ensemble, GpuAdjoint, GpuLes, abi, fields as FL, synthetic_case
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


BOX = ((2, 20), (2, 20), (2, 10))


def _halo_read(g, adj, tmp):
    L = abi.lib()
    buf = np.zeros(L.les_ctx_halo_floats(g.ctx, 0), np.float32)
    abi.check(L.les_ctx_halo_read(g.ctx, 0, buf.ctypes.data))


def _halo_write(g, adj, tmp):
    L = abi.lib()
    buf = np.zeros(L.les_ctx_halo_floats(g.ctx, 0), np.float32)
    abi.check(L.les_ctx_halo_write(g.ctx, 0, buf.ctypes.data))


def _phase_times(g, adj, tmp):
    abi.check(abi.lib().les_ctx_phase_times(g.ctx, 0, (C.c_float * 9)(), 9))


def _reverse(g, adj, tmp):
    adj.zero()
    adj.seed_tke(-1, BOX, 1.0)
    adj.step_b(1, 0)
    adj.read(state=True)


# every call that waits for the step and hands something of it on
CALLS = {
    "sync": lambda g, adj, tmp: g.sync(),
    "metrics": lambda g, adj, tmp: g.metrics(),
    "download": lambda g, adj, tmp: g.download(["u"]),
    "field_sums": lambda g, adj, tmp: g.field_sums(),
    "halo_read": _halo_read,
    "halo_write": _halo_write,
    "phase_times": _phase_times,
    "warmup": lambda g, adj, tmp: g.warmup(1),
    "aveflow_files": lambda g, adj, tmp: g.aveflow(1, 1, 1, 0.0, tmp / "d10", tmp / "d11"),
    "aveflow_download": lambda g, adj, tmp: (g.aveflow(1, 1, 2), g.aveflow_download()),
    "write_restart": lambda g, adj, tmp: g.write_restart(tmp / "d20", tmp / "d21"),
    "adj_tke": lambda g, adj, tmp: adj.tke(-1, BOX),
    "adj_read": _reverse,
}


@pytest.mark.parametrize("call", CALLS)
def test_every_reader_reports_a_void_step(require_gpu, call, tmp_path):
    g = GpuLes(_case((61, 47, 35), 5))
    adj = GpuAdjoint(g, 2, 10)
    try:
        adj.save(0)
        abi.check(abi.lib().les_ctx_set_timing(g.ctx, 2))
        _void(g)
        _times_out(CALLS[call], g, adj, tmp_path)
        g.sync()  # reported once
        assert not list(tmp_path.iterdir()), "files of a void step"
    finally:  # the adjoint before its context
        adj.close()
        g.close()


def test_refined_metrics_report_a_void_step(require_gpu):
    g = GpuLes(_case((62, 48, 35), 5))
    g.warmup(1)
    g.press_refine_fp64(1, 6, 1e-9)
    _void(g)
    _times_out(g.refine_metrics)
    g.close()


def test_an_ensemble_reports_every_void_member(require_gpu):
    gs = [GpuLes(_case((61, 47, 35), 5)), GpuLes(_case((40, 33, 14), 6)), GpuLes(_case((64, 48, 33), 7))]
    for g in gs:
        g.warmup(1)
    for g in (gs[0], gs[2]):
        abi.check(abi.lib().les_ctx_set_sor_wait(g.ctx, 1))
    ens = Ensemble(gs)
    ens.step(1, 1)
    _times_out(ens.sync)
    ens.sync()  # one report for all of them
    for g in gs:
        g.sync()
    ens.close()
    for g in gs:
        g.close()
