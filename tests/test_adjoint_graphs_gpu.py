"""The adjoint's replayed and reverse steps as graphs: the same gradients as
eager launches, also on another starting state and after the plan's scratch
has moved (a larger batch on the same plan), for segments of one step, of an
odd length and of the whole run.

Bound: the states' cotangents of both come from the same kernels in the same
order, so they are equal; the parameter gradients add float partial sums into
doubles by atomics in any order (relative 1e-6 of the vector)."""
import numpy as np
import pytest

from turing_sphere_b200 import (GpuModel, ShtConfig, ShtPlan, defaultParams, mModelByKey,
                                seededNoise)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,every", [("fp32", 1), ("fp32", 5), ("tf32x3", 12)])
def test_graphs_give_the_eager_gradients(device, precision, every):
    lmax, nlat, nphi, steps, batch = 31, 48, 96, 12, 2
    model = mModelByKey("schnakenberg")
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": precision})
    gpu = GpuModel.create(device, plan, model.source, [p.key for p in model.params], model.state,
                          model.species, batch)
    gpu.setParams(defaultParams(model))
    rng = np.random.default_rng(3)
    bar = {s: rng.standard_normal((batch, 2 * plan.nlm)).astype(np.float32) for s in model.state}

    def gradients(seed, graphs):
        gpu.setGraphs(graphs)
        gpu.init(np.concatenate([seededNoise(nlat * nphi, model.seedAmp, seed + k) for k in range(batch)]))
        return gpu.forwardBackward(steps, every, bar)

    want = {seed: gradients(seed, False) for seed in (1, 7)}
    for k, seed in enumerate((1, 7, 1, 7)):
        if k == 2:
            plan.synth(np.zeros(64 * 2 * plan.nlm, dtype=np.float32), 64)  # moves the plan's scratch
        got = gradients(seed, True)
        for s in model.state:
            assert np.array_equal(got[0][s], want[seed][0][s]), (k, s)
        assert np.linalg.norm(got[1] - want[seed][1]) <= 1e-6 * np.linalg.norm(want[seed][1])
    gpu.destroy()
    plan.destroy()
