"""A device without room for the chip-resident SOR's buffers: the step runs on
the passes."""
import pytest

import oracle
from les_halo_b200 import GpuLes, abi, fields as FL, synthetic_case
from tests.helpers import assert_bitexact

pytestmark = pytest.mark.gpu


def test_no_room_keeps_the_passes(require_gpu):
    import torch
    # a domain whose buffers (the words of 64-plane segments, the rhs scratch)
    # take about 20 MB, on a device with 12 MB left
    dims = (257, 203, 61)
    case = synthetic_case(*dims, seed=5, dx=4.0, dy=4.0, masks_and_poisson=oracle.masks_and_poisson)
    ref = GpuLes(case.copy())
    abi.check(abi.lib().les_ctx_set_sor_path(ref.ctx, 1))
    g = GpuLes(case.copy())
    for x in (ref, g):
        x.warmup(1)
    ref.step(1, 2)
    ref.sync()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - (12 << 20), dtype=torch.uint8, device="cuda")
    try:
        g.step(1, 2)
        g.sync()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert_bitexact(g.download(FL.STATE), ref.download(FL.STATE), *dims, FL.STATE)
    assert g.metrics()["sor_iters"] == ref.metrics()["sor_iters"] == 50
    for x in (ref, g):
        x.close()
