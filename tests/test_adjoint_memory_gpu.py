"""A forward/backward call that finds no memory gives back what it had taken:
here 316 MB of checkpoints (256 MiB may stay), before a segment's states (210 GB, more
than the GPU has) are refused; the next call works."""
import numpy as np
import pytest

from turing_sphere_b200 import GpuModel, ShtConfig, ShtPlan, defaultParams, mModelByKey
from turing_sphere_b200._lib import TsError

pytestmark = pytest.mark.gpu


def test_a_call_without_memory_keeps_none(device):
    import torch
    lmax, nlat, nphi = 255, 384, 768
    model = mModelByKey("schnakenberg")
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi))
    gpu = GpuModel.create(device, plan, model.source, [k.key for k in model.params], model.state,
                          model.species, 1)
    gpu.setParams(defaultParams(model))
    bar = {s: np.ones((1, 2 * plan.nlm), dtype=np.float32) for s in model.state}
    gpu.forwardBackward(2, 1, bar)  # the adjoint's own buffers and kernels
    free = torch.cuda.mem_get_info()[0]
    with pytest.raises(TsError, match="out of memory"):
        gpu.forwardBackward(240_000_000, 400_000, bar)
    assert torch.cuda.mem_get_info()[0] >= free - (64 << 20)
    states, params = gpu.forwardBackward(2, 1, bar)
    assert np.isfinite(params).all() and all(np.isfinite(v).all() for v in states.values())
    gpu.destroy()
    plan.destroy()
