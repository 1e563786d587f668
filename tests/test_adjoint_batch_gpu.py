"""The gradient of an instance does not depend on how many instances stand
beside it: the adjoint of a tensor-core plan takes the same Legendre kernels
for two instances as for 65 (more than any batch the FP32 products take).

The Brusselator near its steady state, where the derivative to dt sums a rate
of change that is a difference of terms some 100 times as large.

Bounds: forward and reverse steps run the same kernels field by field, so the
states' cotangents are equal; parameter gradients add the same float partial
sums into doubles in any order (1e-12).  A step compiled otherwise, with its
rounding of 6e-8, would show as 6e-5, another Legendre kernel as 1e-4."""
import numpy as np
import pytest

from turing_sphere_b200 import (GpuModel, ShtConfig, ShtPlan, defaultParams, mModelByKey)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,nlat,nphi,steps,every",
                         [(63, 96, 192, 8, 8), (127, 192, 384, 4, 2), (127, 192, 384, 8, 3)])
def test_gradients_of_two_and_of_many_instances(device, lmax, nlat, nphi, steps, every):
    model = mModelByKey("brusselator")
    p = defaultParams(model)
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": "tf32x3"})
    rng = np.random.default_rng(lmax)
    l_of = np.concatenate([np.arange(m, lmax + 1) for m in range(lmax + 1)])

    def spectra():
        q = rng.standard_normal((65, plan.nlm, 2)) / (l_of[:, None] + 1.0)
        q[:, :lmax + 1, 1] = 0.0  # m = 0
        return q.astype(np.float32)

    start = {}
    for name, mean in (("U", p["A"]), ("V", p["B"] / p["A"])):
        q = 0.1 * spectra()
        q[:, 0, 0] = np.sqrt(4 * np.pi) * mean
        start[name] = q.reshape(65, -1)
    bar = {name: spectra().reshape(65, -1) for name in model.state}
    got = []
    for batch in (2, 65):
        gpu = GpuModel.create(device, plan, model.source, [k.key for k in model.params], model.state,
                              model.species, batch)
        gpu.setParams(p)
        for name in model.state:
            gpu.upload(name, start[name][:batch])
        states, params = gpu.forwardBackward(steps, every, {s: bar[s][:batch] for s in bar})
        got.append(({s: states[s][:2] for s in states}, params[:2]))
        gpu.destroy()
    for s in model.state:
        assert np.array_equal(got[0][0][s], got[1][0][s]), s
    assert np.linalg.norm(got[0][1] - got[1][1]) <= 1e-12 * np.linalg.norm(got[1][1])
    plan.destroy()
