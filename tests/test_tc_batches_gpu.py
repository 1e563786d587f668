"""The tensor-core contraction on batches that take it: 65 device fields (two
blocks of 64, more than any batch of the FP32 products) on the grids, tiles
and plan kinds of the single-field tests, which a tensor-core plan now runs
as FP32 products.  Every field is the first one times a power of two and so
is its result, bit by bit; the first is checked against the f64 oracle
(relative L2 <= 1e-5), and differs in some bit from the same field in a batch
of the products, which shows that another kernel ran."""
import numpy as np
import pytest

from oracle import oracle as O
from turing_sphere_b200 import GpuModel, ShtConfig, ShtPlan, defaultParams, mModelByKey
from turing_sphere_b200._lib import TS_ERR_TIMEOUT, TsError

from .test_sht_gpu import scaled_spectrum

pytestmark = pytest.mark.gpu

TOL = 1e-5
BATCH = 65


def transform(device, plan, name, x, n, batch):
    import torch
    scale = np.ldexp(np.float32(1), -(np.arange(batch) % 5)).astype(np.float32)[:, None]
    src = torch.from_numpy(scale * x[None, :]).cuda()
    out = torch.full((batch, n), float("nan"), device="cuda")
    torch.cuda.synchronize()
    getattr(plan, name)(src.data_ptr(), out.data_ptr(), batch)
    device.sync()
    assert torch.equal(out, torch.from_numpy(scale).cuda() * out[0])
    return out[0].cpu().numpy()


def check(device, parity, plan, label, lmax, mmax, nlat, nphi, q, from_lm=0):
    ref = O.ShtReference(lmax, mmax, nlat, nphi)
    s64 = ref.synth(q.astype(np.float64))
    s32 = s64.astype(np.float32)
    q64 = ref.analys(s32.astype(np.float64))
    syn = transform(device, plan, "synth_dev", q, s64.size, BATCH)
    ana = transform(device, plan, "analys_dev", s32, q.size, BATCH)
    plan.status()
    parity(f"contraction {label} synth", O.rel_l2(syn, s64), TOL)
    parity(f"contraction {label} analys", O.rel_l2(ana[from_lm:], q64[from_lm:]), TOL)
    assert not np.array_equal(syn, transform(device, plan, "synth_dev", q, s64.size, 4))
    assert not np.array_equal(ana, transform(device, plan, "analys_dev", s32, q.size, 4))


@pytest.mark.parametrize("lmax,nlat,nphi,mmax", [(15, 16, 32, 15), (31, 32, 64, 31), (31, 33, 64, 31),
                                                 (40, 48, 96, 20), (63, 96, 192, 63), (255, 384, 768, 255),
                                                 (511, 768, 1536, 511), (1023, 1536, 3072, 1023)])
def test_contraction_parity(device, parity, lmax, nlat, nphi, mmax):
    plan = ShtPlan.create(device, ShtConfig(lmax, mmax, nlat, nphi), {"precision": "tf32x3"})
    check(device, parity, plan, f"lmax{lmax} mmax{mmax} nlat{nlat}", lmax, mmax, nlat, nphi,
          scaled_spectrum(lmax, mmax, 21))
    plan.destroy()


@pytest.mark.parametrize("lmax,nlat,nphi", [(255, 384, 768), (511, 768, 1536)])
def test_polar_skip_of_the_contraction(device, parity, lmax, nlat, nphi):
    """Orders from lmax / 2 on, the only ones that the skip touches."""
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": "tf32x3"})
    assert plan.shapes["tc_skip_tiles"] > 0 and plan.shapes["tc_skip_chunks"] > 0
    m0 = lmax // 2
    start = 2 * (m0 * (lmax + 1) - m0 * (m0 - 1) // 2)
    q = scaled_spectrum(lmax, lmax, 31)
    q[:start] = 0
    check(device, parity, plan, f"lmax{lmax} polar skip", lmax, lmax, nlat, nphi, q, start)
    plan.destroy()


def test_tuned_tiles_of_the_contraction(device, parity):
    lmax, nlat, nphi = 127, 192, 384
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": "tf32x3", "autotune": True})
    assert plan.shapes["tuned"]
    check(device, parity, plan, "lmax127 autotuned", lmax, lmax, nlat, nphi, scaled_spectrum(lmax, lmax, 32))
    plan.destroy()


def test_the_contraction_recovers_from_a_timeout(device, parity):
    """The same kernels after their bounded waits ran out (the stall hook)."""
    lmax, nlat, nphi = 31, 32, 64
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": "tf32x3"})
    q = scaled_spectrum(lmax, lmax, 7)
    plan.testStall(True, wait_limit=4096)
    plan.synth(np.tile(q, (BATCH, 1)), batch=BATCH)
    with pytest.raises(TsError) as ei:
        plan.status()
    assert ei.value.status == TS_ERR_TIMEOUT
    plan.testStall(False)
    check(device, parity, plan, "lmax31 after a timeout", lmax, lmax, nlat, nphi, q)
    plan.destroy()


def test_fused_epilogue_of_the_contraction(device, parity):
    """A model of few instances whose grid is too tall for the products'
    tables (over 2 GB): the tensor-core analysis with the update in its
    epilogue (four launches a step), two steps against the oracle."""
    lmax, nlat, nphi, steps = 511, 8192, 1536, 2
    model = mModelByKey("schnakenberg")
    p = defaultParams(model)
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": "tf32x3"})
    gpu = GpuModel.create(device, plan, model.source, [k.key for k in model.params], model.state,
                          model.species, 1)
    assert gpu.counts("step") == (5, 4)
    gpu.setParams(p)
    st0 = []
    for name, mean in (("U", p["a"] + p["b"]), ("V", p["b"] / (p["a"] + p["b"]) ** 2)):
        q = 0.1 * scaled_spectrum(lmax, lmax, len(st0))
        q[0] = np.sqrt(4 * np.pi) * mean
        st0.append(q)
        gpu.upload(name, q)
    gpu.step(steps)
    want = O.ShtReference(lmax, lmax, nlat, nphi).model_step(
        "schnakenberg", [np.float32(p[k.key]) for k in model.params], np.stack(st0).astype(np.float64), steps)
    plan.status()
    for i, name in enumerate(model.state):
        parity(f"tf32x3 fused epilogue lmax511 nlat8192 {name}", O.rel_l2(gpu.read(name), want[i]), 1e-4)
    gpu.destroy()
    plan.destroy()
