"""The momentum kernels' tiles at their edges: pieces of the k march, edge
tiles of uniform grids (spacings that are and are not powers of two) and of
stretched ones, against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
from les_halo_b200 import GpuLes, fields as FL, synthetic_case

pytestmark = pytest.mark.gpu


def _case(ip, jp, kp, dx, stretch):
    def stretched(case, zbm):
        # before masks_and_poisson reads the metrics
        if stretch:
            A = case.arrays
            A["dx1"][:] = (dx * (1 + 0.1 * np.sin(np.arange(A["dx1"].size)))).astype(np.float32)
            A["dy1"][:] = (dx * (1 + 0.1 * np.cos(np.arange(A["dy1"].size)))).astype(np.float32)
            A["dxs"][:] = A["dx1"][1:-1] / np.float32(2) + A["dx1"][2:] / np.float32(2)
            A["dys"][:] = A["dy1"][:-1] / np.float32(2) + A["dy1"][1:] / np.float32(2)
        oracle.masks_and_poisson(case, zbm)

    return synthetic_case(ip, jp, kp, seed=3, masks_and_poisson=stretched, dx=dx, dy=dx)


# one tile with one cell past it, exact tiles, a last tile of one column or
# row, the shortest band, heights that cut into pieces of unequal length
@pytest.mark.parametrize("ip,jp,kp", [(33, 9, 3), (32, 16, 7), (65, 12, 19), (31, 25, 40), (40, 11, 5)])
@pytest.mark.parametrize("dx,stretch", [(4.0, False), (20.0, False), (5.0, True)])
def test_tile_edges_bitexact(ip, jp, kp, dx, stretch):
    ref = _case(ip, jp, kp, dx, stretch)
    gpu = GpuLes(ref.copy())
    oracle.ifdata(ref, 1)
    gpu.warmup(1)
    oracle.run_steps(ref, 1, 3)
    gpu.step(1, 3)
    got = gpu.download(FL.STATE)
    gpu.close()
    for n in FL.STATE:
        assert np.array_equal(got[n].view(np.uint32), ref.a(n).view(np.uint32)), n
