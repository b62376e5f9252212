"""Grids whose SOR is one launch, on the SOR passes instead: the passes' small
odd-jp grids and their shapes inside an ensemble, and which of the two runs."""
import ctypes as C

import numpy as np
import pytest

import oracle
from les_halo_b200 import Ensemble, GpuLes, abi, fields as FL, synthetic_case
from tests.helpers import assert_bitexact

pytestmark = pytest.mark.gpu
ALL = FL.STATE + FL.MASKS


def _case(dims, seed, **kw):
    return synthetic_case(*dims, seed=seed, masks_and_poisson=oracle.masks_and_poisson, **kw)


def _passes(case):
    g = GpuLes(case)
    abi.check(abi.lib().les_ctx_set_sor_resident(g.ctx, 0))
    g.warmup(1)
    return g


def _iters_per_pass(g):
    t, ty = C.c_int(), C.c_int()
    abi.check(abi.lib().les_ctx_sor_tile(g.ctx, C.byref(t), C.byref(ty)))
    return t.value


# 9 rows: the 8-row region of the shortest pass shape holds 8 of them
@pytest.mark.parametrize("dims", [(70, 33, 10), (40, 9, 12)])
def test_odd_jp_passes_against_oracle(require_gpu, dims):
    ref = _case(dims, sum(dims))
    gpu = _passes(ref.copy())
    oracle.ifdata(ref, 1)
    for n in range(1, 4):
        iters = oracle.run_steps(ref, n, 1)
        gpu.step(n, 1)
        assert gpu.metrics()["sor_iters"] == iters[0]
    assert not abi.lib().les_ctx_sor_resident(gpu.ctx) and _iters_per_pass(gpu) == 1
    assert_bitexact(gpu.download(FL.STATE), {k: ref.a(k) for k in FL.STATE}, *dims, FL.STATE)
    gpu.close()


def test_ensemble_on_tuned_passes_equals_colour_sweeps(require_gpu):
    doms = [((24, 20, 12), 3), ((40, 26, 16), 4), ((17, 15, 9), 5), ((33, 18, 10), 6)]
    cases = [_case(*d) for d in doms]
    solo, members = [GpuLes(c.copy()) for c in cases], [_passes(c.copy()) for c in cases]
    for g in solo:
        abi.check(abi.lib().les_ctx_set_sor_path(g.ctx, 1))
        g.warmup(1)
    ens = Ensemble(members)
    ens.step(1, 4)
    assert all(_iters_per_pass(g) > 0 for g in members)
    for g in solo:
        g.step(1, 4)
    for (d, _), a, b in zip(doms, members, solo):
        assert_bitexact(a.download(ALL), b.download(ALL), *d, ALL)
        assert a.metrics()["sor_iters"] == b.metrics()["sor_iters"]
    ens.close()
    for g in solo + members:
        g.close()


def test_which_sor_runs(require_gpu):
    L, dims = abi.lib(), (61, 47, 35)
    g = GpuLes(_case(dims, 5, dx=4.0, dy=4.0))
    g.warmup(1)
    n = []
    for on in (1, 0, 1):
        abi.check(L.les_ctx_set_sor_resident(g.ctx, on))
        n0 = g.launches()
        g.step(2, 1)
        n.append(g.launches() - n0)
        assert L.les_ctx_sor_resident(g.ctx) == on
    assert n[0] == n[2] < 24 < n[1]
    abi.check(L.les_ctx_set_sor_path(g.ctx, 1))
    assert L.les_ctx_sor_resident(g.ctx) == 0
    assert np.isfinite(g.metrics()["sor"])
    g.close()
