"""The adjoint's graphs run on a fresh plan and model from their first call
on: each kind of step is eager twice and a graph from then on, whatever the
lengths of the segments; the gradients are those of eager launches on another
fresh model (equal states' cotangents; parameter gradients add the same float
partial sums into doubles in any order, 1e-12)."""
import ctypes as C

import numpy as np
import pytest

from turing_sphere_b200 import (GpuModel, ShtConfig, ShtPlan, _lib, defaultParams, mModelByKey,
                                seededNoise)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "tf32x3"])
@pytest.mark.parametrize("steps,every", [(16, 8), (9, 4), (6, 1), (7, 20)])
def test_both_graphs_run_on_a_fresh_model(device, precision, steps, every):
    lmax, nlat, nphi, batch = 31, 48, 96, 2
    model = mModelByKey("schnakenberg")

    def fresh(graphs):
        plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": precision})
        gpu = GpuModel.create(device, plan, model.source, [p.key for p in model.params], model.state,
                              model.species, batch)
        gpu.setParams(defaultParams(model))
        gpu.setGraphs(graphs)
        gpu.init(np.concatenate([seededNoise(nlat * nphi, model.seedAmp, 1 + k) for k in range(batch)]))
        rng = np.random.default_rng(3)
        bar = {s: rng.standard_normal((batch, 2 * plan.nlm)).astype(np.float32) for s in model.state}
        got = gpu.forwardBackward(steps, every, bar)
        n = C.c_long(), C.c_long()
        _lib.check(_lib.lib().ts_model_adjoint_graphs(gpu.handle, C.byref(n[0]), C.byref(n[1])))
        gpu.destroy()
        plan.destroy()
        return got, n[0].value, n[1].value

    want, replayed, reverse = fresh(False)
    assert (replayed, reverse) == (0, 0)
    got, replayed, reverse = fresh(True)
    segments = -(-steps // every)
    assert replayed == max(0, steps - segments - 2)
    assert reverse == steps - 2
    for s in model.state:
        assert np.array_equal(got[0][s], want[0][s]), s
    assert np.linalg.norm(got[1] - want[1]) <= 1e-12 * np.linalg.norm(want[1])
