"""The momentum kernels' k march in pieces of several planes that end below the
top one: pieces of 2, 3, 7 and all planes, with last pieces of one plane and
more, on the tiles of uniform and stretched grids, against the oracle."""
import numpy as np
import pytest

import oracle
from les_halo_b200 import GpuLes, abi, fields as FL, synthetic_case

pytestmark = pytest.mark.gpu


def _case(ip, jp, kp, dx, stretch):
    def masks(case, zbm):
        if stretch:
            A = case.arrays
            A["dx1"][:] = (dx * (1 + 0.1 * np.sin(np.arange(A["dx1"].size)))).astype(np.float32)
            A["dy1"][:] = (dx * (1 + 0.1 * np.cos(np.arange(A["dy1"].size)))).astype(np.float32)
            A["dxs"][:] = A["dx1"][1:-1] / np.float32(2) + A["dx1"][2:] / np.float32(2)
            A["dys"][:] = A["dy1"][:-1] / np.float32(2) + A["dy1"][1:] / np.float32(2)
        oracle.masks_and_poisson(case, zbm)

    return synthetic_case(ip, jp, kp, seed=3, masks_and_poisson=masks, dx=dx, dy=dx)


# (jp = 11 and less: no staged band); 15 = 7 * 2 + 1 = 2 * 7 + 1, 16 = 5 * 3 + 1
@pytest.mark.parametrize("ip,jp,kp", [(33, 13, 15), (65, 25, 16), (40, 11, 15), (96, 48, 40)])
@pytest.mark.parametrize("dx,stretch", [(4.0, False), (20.0, False), (5.0, True)])
def test_pieces_bitexact(require_gpu, ip, jp, kp, dx, stretch):
    ref = _case(ip, jp, kp, dx, stretch)
    start = ref.copy()
    oracle.ifdata(ref, 1)
    oracle.run_steps(ref, 1, 3)
    for planes in (2, 3, 7, kp):
        gpu = GpuLes(start.copy())
        abi.check(abi.lib().les_ctx_set_mom_planes(gpu.ctx, planes))
        gpu.warmup(1)
        gpu.step(1, 3)
        got = gpu.download(FL.STATE)
        gpu.close()
        for n in FL.STATE:
            assert np.array_equal(got[n].view(np.uint32), ref.a(n).view(np.uint32)), (planes, n)
