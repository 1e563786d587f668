"""A tensor-core plan that has no memory for the FP32 products' tables when a
small batch first wants them stays with the contraction: the call succeeds
and no later one tries the allocation again."""
import contextlib

import numpy as np
import pytest

from oracle import oracle as O
from turing_sphere_b200 import ShtConfig, ShtPlan

from .test_leg_gemm_gpu import spectrum

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def little_memory(left):
    """All but `left` bytes of the GPU's free memory taken for the block."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    ballast = [torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")]
    try:
        yield
    finally:
        ballast.clear()
        torch.cuda.empty_cache()


def test_no_memory_for_the_tables(device, parity):
    import torch
    lmax, nlat, nphi = 511, 768, 1536  # 415 MB of tables
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": "tf32x3"})
    q = spectrum(lmax, lmax, 1)
    src = torch.from_numpy(np.tile(q, (64, 1))).cuda()
    grid = torch.empty(64, nlat * nphi, device="cuda")
    torch.cuda.synchronize()
    plan.synth_dev(src.data_ptr(), grid.data_ptr(), 64)  # the contraction: its image and the scratch
    grid.zero_()
    with little_memory(256 << 20):
        plan.synth_dev(src.data_ptr(), grid.data_ptr(), 4)
        device.sync()
    first = grid[:4].clone()
    parity("tf32x3 lmax511 B4 synth without tables", O.rel_l2(
        first[3].cpu().numpy(), O.ShtReference(lmax, lmax, nlat, nphi).synth(q.astype(np.float64))), 1e-5)
    free = torch.cuda.mem_get_info()[0]
    grid.zero_()
    torch.cuda.synchronize()
    plan.synth_dev(src.data_ptr(), grid.data_ptr(), 4)
    device.sync()
    assert torch.cuda.mem_get_info()[0] == free
    assert torch.equal(grid[:4], first)
    plan.destroy()


def test_no_memory_for_the_scratch(device, parity):
    """With the tables made and the operand image in place, a small analysis
    that finds no memory for the products' scratch (50 MB) runs as the
    contraction."""
    import torch
    lmax, nlat, nphi = 511, 768, 1536
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": "tf32x3"})
    ref = O.ShtReference(lmax, lmax, nlat, nphi)
    q = spectrum(lmax, lmax, 2)
    grid = ref.synth(q.astype(np.float64)).astype(np.float32)
    spat = torch.from_numpy(np.tile(grid, (64, 1))).cuda()
    spec = torch.from_numpy(np.tile(q, (64, 1))).cuda()
    fm = torch.empty(4, (lmax + 1) * nlat * 2, device="cuda")
    torch.cuda.synchronize()
    plan.stage_dev("legSynth", spec.data_ptr(), fm.data_ptr(), 4)    # the tables
    plan.analys_dev(spat.data_ptr(), spec.data_ptr(), 64)            # the image
    with little_memory(24 << 20):
        plan.analys_dev(spat.data_ptr(), spec.data_ptr(), 4)
        device.sync()
    parity("tf32x3 lmax511 B4 analys without scratch",
           O.rel_l2(spec[3].cpu().numpy(), ref.analys(grid.astype(np.float64))), 1e-5)
    plan.destroy()
