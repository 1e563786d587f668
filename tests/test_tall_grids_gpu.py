"""Grids with many latitudes, where the shared memory of the kernels for one
and two fields (16 bytes a northern latitude and field) comes to its limits."""
import numpy as np
import pytest

from oracle import oracle as O
from turing_sphere_b200 import (GpuModel, ShtConfig, ShtPlan, defaultParams, mModelByKey,
                                seededNoise)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "tf32x3"])
@pytest.mark.parametrize("nlat", [1024, 2047, 2048])
def test_one_instance_of_two_species(device, parity, precision, nlat):
    """At 2047 and 2048 latitudes the analysis asks for exactly 48 KB beside
    its static shared memory.  Three steps against the oracle (the relative L2
    bound of the model tests, 1e-4)."""
    lmax, nphi, steps = 31, 64, 3
    model = mModelByKey("schnakenberg")
    p = defaultParams(model)
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": precision})
    gpu = GpuModel.create(device, plan, model.source, [k.key for k in model.params], model.state,
                          model.species, 1)
    gpu.setParams(p)
    gpu.init(seededNoise(nlat * nphi, model.seedAmp, 1))
    st0 = [gpu.read(s) for s in model.state]
    gpu.step(steps)
    want = O.ShtReference(lmax, lmax, nlat, nphi).model_step(
        "schnakenberg", [np.float32(p[k.key]) for k in model.params], np.stack(st0).astype(np.float64), steps)
    for i, name in enumerate(model.state):
        parity(f"{precision} schnakenberg lmax31 nlat{nlat} {name}", O.rel_l2(gpu.read(name), want[i]), 1e-4)
    gpu.destroy()
    plan.destroy()


@pytest.mark.parametrize("precision", ["fp32", "tf32x3"])
@pytest.mark.parametrize("nlat,batch", [(13440, 2), (13600, 2), (28000, 1), (28201, 1), (28201, 2)])
def test_few_fields_beyond_the_shared_memory(device, parity, precision, nlat, batch):
    """Either side of the most latitudes whose columns fit in shared memory:
    the analysis against the oracle (1e-5, the transforms' bound)."""
    import torch
    lmax, nphi = 31, 64
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": precision})
    grid = np.random.default_rng(nlat).standard_normal((batch, nlat * nphi)).astype(np.float32)
    src, out = torch.from_numpy(grid).cuda(), torch.empty(batch, 2 * plan.nlm, device="cuda")
    torch.cuda.synchronize()
    plan.analys_dev(src.data_ptr(), out.data_ptr(), batch)
    device.sync()
    ref = O.ShtReference(lmax, lmax, nlat, nphi)
    for f in range(batch):
        want = ref.analys(grid[f].astype(np.float64))
        parity(f"{precision} lmax31 nlat{nlat} B{batch} analys {f}", O.rel_l2(out[f].cpu().numpy(), want), 1e-5)
    plan.destroy()


def test_one_instance_beyond_the_shared_memory(device, parity):
    """A two-species model on 13600 latitudes takes the tiled analysis."""
    lmax, nlat, nphi, steps = 31, 13600, 64, 2
    model = mModelByKey("schnakenberg")
    p = defaultParams(model)
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi))
    gpu = GpuModel.create(device, plan, model.source, [k.key for k in model.params], model.state,
                          model.species, 1)
    gpu.setParams(p)
    gpu.init(seededNoise(nlat * nphi, model.seedAmp, 1))
    st0 = [gpu.read(s) for s in model.state]
    gpu.step(steps)
    want = O.ShtReference(lmax, lmax, nlat, nphi).model_step(
        "schnakenberg", [np.float32(p[k.key]) for k in model.params], np.stack(st0).astype(np.float64), steps)
    for i, name in enumerate(model.state):
        parity(f"fp32 schnakenberg lmax31 nlat13600 {name}", O.rel_l2(gpu.read(name), want[i]), 1e-4)
    gpu.destroy()
    plan.destroy()


@pytest.mark.parametrize("lmax,nlat", [(3, 641), (3, 670), (3, 770), (3, 1566), (1, 3074), (1, 3134)])
def test_recurrence_analysis_between_its_shapes(device, parity, lmax, nlat):
    """Northern latitudes between the recurrence kernel's shapes (grids small
    enough in lmax to take it): one and three fields against the oracle."""
    import torch
    nphi = 32
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi))
    ref = O.ShtReference(lmax, lmax, nlat, nphi)
    for batch in (1, 3):
        grid = np.random.default_rng(nlat).standard_normal((batch, nlat * nphi)).astype(np.float32)
        src, out = torch.from_numpy(grid).cuda(), torch.empty(batch, 2 * plan.nlm, device="cuda")
        torch.cuda.synchronize()
        plan.analys_dev(src.data_ptr(), out.data_ptr(), batch)
        device.sync()
        for f in range(batch):
            want = ref.analys(grid[f].astype(np.float64))
            parity(f"fp32 lmax{lmax} nlat{nlat} B{batch} analys {f}", O.rel_l2(out[f].cpu().numpy(), want), 1e-5)
    plan.destroy()
