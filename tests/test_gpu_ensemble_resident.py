"""Ensembles of members whose SOR is one launch and members on SOR passes."""
import ctypes as C

import numpy as np
import pytest

import oracle
from les_halo_b200 import Ensemble, GpuLes, abi, fields as FL, synthetic_case
from tests.helpers import assert_bitexact

pytestmark = pytest.mark.gpu
ALL = FL.STATE + FL.MASKS


def _case(dims, seed, stretch=False):
    def masks(case, zbm):
        if stretch:  # x spacings that differ keep a grid on the passes
            A = case.arrays
            A["dx1"][:] = (4 * (1 + 0.1 * np.sin(np.arange(A["dx1"].size)))).astype(np.float32)
            A["dxs"][:] = A["dx1"][1:-1] / np.float32(2) + A["dx1"][2:] / np.float32(2)
        oracle.masks_and_poisson(case, zbm)

    return synthetic_case(*dims, seed=seed, dx=4.0, dy=4.0, masks_and_poisson=masks)


def _iters_per_pass(g):
    t, ty = C.c_int(), C.c_int()
    abi.check(abi.lib().les_ctx_sor_tile(g.ctx, C.byref(t), C.byref(ty)))
    return t.value


def test_the_tuner_times_only_members_that_launch_passes(require_gpu):
    doms = [(64, 48, 24), (61, 47, 35), (40, 26, 16)]
    cases = [_case(d, s, stretch=s == 0) for s, d in enumerate(doms)]
    solo, members = [GpuLes(c.copy()) for c in cases], [GpuLes(c.copy()) for c in cases]
    for g in solo + members:
        g.warmup(1)
    n0 = members[1].launches()
    ens = Ensemble(members)
    ens.step(1, 3)
    assert _iters_per_pass(members[0]) > 0
    assert [_iters_per_pass(g) for g in members[1:]] == [0, 0], "tuned for passes that no step launches"
    assert members[1].launches() == n0
    for g in solo:
        g.step(1, 3)
    for d, a, b in zip(doms, members, solo):
        assert_bitexact(a.download(ALL), b.download(ALL), *d, ALL)
    ens.close()
    for g in solo + members:
        g.close()
