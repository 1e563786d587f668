"""The batched FP32 Legendre products (kernels/leg_gemm.cuh) at the sizes where
their tiles end: 16-degree k-tiles, blocks of 8, 16, 24 and 32 degrees (one or
two to a parity, one or two CTAs to an order), 64-latitude tiles, 8-, 16- and
32-field tiles, odd latitudes, mmax < lmax.

Every field is the first one times a power of two, so its result has to be
the first one's times that power, bit by bit; the first one is checked against
the f64 oracle (relative L2 <= 1e-5, the plain FP32 path's bound up to lmax 255).
"""
import numpy as np
import pytest

from oracle import oracle as O
from turing_sphere_b200 import (GpuModel, ShtConfig, ShtPlan, defaultParams, mModelByKey,
                                seededNoise)

pytestmark = pytest.mark.gpu

TOL = 1e-5
CASES = [
    (31, 31, 48, 96, 8), (31, 31, 33, 64, 9), (62, 62, 96, 192, 33), (64, 50, 131, 256, 17),
    (95, 95, 128, 256, 16), (127, 127, 192, 384, 5), (128, 100, 193, 512, 36),
    (129, 129, 260, 512, 16), (190, 190, 320, 768, 4), (255, 255, 384, 768, 4),
    (255, 3, 384, 768, 70),
]


def spectrum(lmax, mmax, seed):
    q = np.random.default_rng(seed).standard_normal((O.nlm_calc(lmax, mmax), 2))
    l_of = np.concatenate([np.arange(m, lmax + 1) for m in range(mmax + 1)])
    q /= l_of[:, None] + 1.0
    q[:lmax + 1, 1] = 0.0  # m = 0
    return q.astype(np.float32).ravel()


@pytest.mark.parametrize("lmax,mmax,nlat,nphi,batch", CASES)
def test_every_field_of_a_batch(device, parity, lmax, mmax, nlat, nphi, batch):
    import torch
    plan = ShtPlan.create(device, ShtConfig(lmax, mmax, nlat, nphi))
    ref = O.ShtReference(lmax, mmax, nlat, nphi)

    def run(call, x, n):  # one call on device arrays (host arrays go in chunks of fields)
        src = torch.from_numpy(x).cuda()
        dst = torch.empty(batch, n, device="cuda")
        torch.cuda.synchronize()
        call(src.data_ptr(), dst.data_ptr(), batch)
        device.sync()
        return dst.cpu().numpy()

    scale = np.ldexp(np.float32(1), -(np.arange(batch) % 5)).astype(np.float32)[:, None]
    q = spectrum(lmax, mmax, lmax + batch)
    grid = run(plan.synth_dev, scale * q[None, :], nlat * nphi)
    want = ref.synth(q.astype(np.float64))
    parity(f"leg_gemm synth lmax{lmax} mmax{mmax} nlat{nlat} B{batch}", O.rel_l2(grid[0], want), TOL)
    assert np.array_equal(grid, scale * grid[0])
    g = want.astype(np.float32)
    back = run(plan.analys_dev, scale * g[None, :].reshape(1, -1), q.size)
    parity(f"leg_gemm analys lmax{lmax} mmax{mmax} nlat{nlat} B{batch}",
           O.rel_l2(back[0], ref.analys(g.astype(np.float64))), TOL)
    assert np.array_equal(back, scale * back[0])
    plan.destroy()


def test_first_call_under_capture(device):
    """A plan's first calls can be captured: they allocate nothing, and the
    replay gives the bits of a call outside the capture."""
    import torch
    lmax, nlat, nphi, batch = 63, 96, 192, 16
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi))
    q = torch.from_numpy(np.stack([spectrum(lmax, lmax, k) for k in range(batch)])).cuda()
    fm = torch.zeros(2, batch, (lmax + 1) * nlat * 2, device="cuda")
    out = torch.zeros(2, batch, q.shape[1], device="cuda")
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        plan.stage_dev("legSynth", q.data_ptr(), fm[0].data_ptr(), batch, stream.cuda_stream)
        plan.stage_dev("legAnalys", fm[0].data_ptr(), out[0].data_ptr(), batch, stream.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    plan.stage_dev("legSynth", q.data_ptr(), fm[1].data_ptr(), batch)
    plan.stage_dev("legAnalys", fm[0].data_ptr(), out[1].data_ptr(), batch)
    device.sync()
    assert torch.equal(fm[0], fm[1]) and torch.equal(out[0], out[1])
    plan.destroy()


def test_model_of_many_instances(device, parity):
    """A batched FP32 model (the update in the epilogue of the products)
    against the oracle and the launches it counts."""
    lmax, nlat, nphi, batch, steps = 63, 96, 192, 9, 20
    model = mModelByKey("schnakenberg")
    p = defaultParams(model)
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi))
    gpu = GpuModel.create(device, plan, model.source, [k.key for k in model.params], model.state,
                          model.species, batch)
    sets = [dict(p, D1=p["D1"] * (1 + 0.1 * k)) for k in range(batch)]
    gpu.setParams(sets)
    assert gpu.counts("step") == (5, 3)
    gpu.init(np.concatenate([seededNoise(nlat * nphi, model.seedAmp, 1 + k) for k in range(batch)]))
    st0 = [gpu.read(s) for s in model.state]
    gpu.step(steps)
    st = [gpu.read(s) for s in model.state]
    ref = O.ShtReference(lmax, lmax, nlat, nphi)
    for k in (0, batch - 1):
        prm = [np.float32(sets[k][x.key]) for x in model.params]
        want = ref.model_step("schnakenberg", prm, np.stack([s[k] for s in st0]).astype(np.float64), steps)
        for i, name in enumerate(model.state):
            parity(f"batched fp32 schnakenberg lmax63 {steps} steps inst{k} {name}",
                   O.rel_l2(st[i][k], want[i]), 1e-4)
    gpu.destroy()
    plan.destroy()


# (lmax, mmax, nlat, nphi, batch): on a tensor-core plan the largest batches of
# the products and the smallest of the contraction, on grids whose tables lie
# on either side of 2 and 64 MB, with odd latitudes and mmax < lmax
TC_CASES = [(63, 63, 96, 192, 48), (63, 63, 96, 192, 49), (100, 90, 151, 512, 16),
            (100, 90, 151, 512, 17), (170, 150, 257, 512, 48), (170, 150, 257, 512, 65),
            (255, 255, 384, 768, 1), (319, 319, 640, 1536, 33)]


@pytest.mark.parametrize("lmax,mmax,nlat,nphi,batch", TC_CASES)
def test_batches_of_a_tensor_core_plan(device, parity, lmax, mmax, nlat, nphi, batch):
    """Every field of both routes against the f64 oracle's transform of the
    first one (relative L2 <= 1e-5: the bar of both plans' transforms)."""
    import torch
    plan = ShtPlan.create(device, ShtConfig(lmax, mmax, nlat, nphi), {"precision": "tf32x3"})
    ref = O.ShtReference(lmax, mmax, nlat, nphi)
    scale = np.ldexp(np.float32(1), -(np.arange(batch) % 5)).astype(np.float32)[:, None]
    q = spectrum(lmax, mmax, lmax + batch)
    want = ref.synth(q.astype(np.float64))
    g = want.astype(np.float32)
    worst = [0.0, 0.0]
    for k, (call, x, y) in enumerate(((plan.synth_dev, q, want),
                                      (plan.analys_dev, g, ref.analys(g.astype(np.float64))))):
        src = torch.from_numpy(scale * x[None, :]).cuda()
        dst = torch.empty(batch, y.size, device="cuda")
        torch.cuda.synchronize()
        call(src.data_ptr(), dst.data_ptr(), batch)
        device.sync()
        got = dst.cpu().numpy() / scale
        worst[k] = max(O.rel_l2(got[f], y) for f in range(batch))
    plan.status()
    parity(f"tf32x3 lmax{lmax} mmax{mmax} nlat{nlat} B{batch} synth", worst[0], TOL)
    parity(f"tf32x3 lmax{lmax} mmax{mmax} nlat{nlat} B{batch} analys", worst[1], TOL)
    plan.destroy()


@pytest.mark.parametrize("precision", ["fp32", "tf32x3"])
@pytest.mark.parametrize("lmax,mmax,nlat,nphi", [(63, 63, 96, 192), (64, 60, 131, 256), (97, 97, 100, 256),
                                                 (130, 130, 263, 768), (255, 255, 384, 768)])
def test_one_and_two_fields(device, parity, precision, lmax, mmax, nlat, nphi):
    """The kernels without staging: rows of 16, 32 and 64 degrees, one and two
    CTAs to an order, odd latitudes; both fields against the oracle."""
    import torch
    plan = ShtPlan.create(device, ShtConfig(lmax, mmax, nlat, nphi), {"precision": precision})
    ref = O.ShtReference(lmax, mmax, nlat, nphi)
    q = np.stack([spectrum(lmax, mmax, 5 + k) for k in range(2)])
    want = np.stack([ref.synth(x.astype(np.float64)) for x in q])
    g = want.astype(np.float32)
    back = np.stack([ref.analys(x.astype(np.float64)) for x in g])
    for batch in (1, 2):
        for name, call, x, y in (("synth", plan.synth_dev, q, want), ("analys", plan.analys_dev, g, back)):
            src = torch.from_numpy(x[2 - batch:]).cuda()
            dst = torch.full((batch, y.shape[1]), float("nan"), device="cuda")
            torch.cuda.synchronize()
            call(src.data_ptr(), dst.data_ptr(), batch)
            device.sync()
            worst = max(O.rel_l2(dst[f].cpu().numpy(), y[2 - batch + f]) for f in range(batch))
            parity(f"{precision} lmax{lmax} mmax{mmax} nlat{nlat} B{batch} {name}", worst, TOL)
    plan.destroy()


@pytest.mark.parametrize("precision", ["fp32", "tf32x3"])
@pytest.mark.parametrize("batch", [1, 4])
def test_a_chain_of_small_calls(device, parity, precision, batch):
    """Calls small enough to launch early (each kernel may start while the one
    before it runs), 200 round trips back to back over two coefficient buffers
    and one grid, then the same chain with a wait after every call: the same
    bits, and the first transform against the oracle."""
    import torch
    lmax, nlat, nphi = 63, 96, 192
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": precision})
    ref = O.ShtReference(lmax, lmax, nlat, nphi)
    q0 = np.stack([spectrum(lmax, lmax, 11 + k) for k in range(batch)])
    grid = torch.empty(batch, nlat * nphi, device="cuda")

    def chain(n, wait):
        a = [torch.from_numpy(q0).cuda(), torch.zeros(q0.shape, device="cuda")]
        torch.cuda.synchronize()
        for i in range(n):
            plan.synth_dev(a[i & 1].data_ptr(), grid.data_ptr(), batch)
            if wait:
                device.sync()
            plan.analys_dev(grid.data_ptr(), a[1 - (i & 1)].data_ptr(), batch)
            if wait:
                device.sync()
        device.sync()
        return a[n & 1].cpu().numpy(), grid.cpu().numpy()

    first = chain(1, True)
    parity(f"{precision} lmax63 B{batch} chain synth", O.rel_l2(first[1][0], ref.synth(q0[0].astype(np.float64))), TOL)
    slow, fast = chain(200, True), chain(200, False)
    assert np.array_equal(slow[0], fast[0]) and np.array_equal(slow[1], fast[1])
    plan.destroy()


@pytest.mark.parametrize("lmax,nlat,nphi", [(319, 640, 1536), (127, 256, 512), (170, 342, 1024)])
def test_contraction_repeats_its_bits_on_grids_of_partial_tiles(device, lmax, nlat, nphi):
    """The tensor-core synthesis where the last latitude tile holds whole chunks
    and then none: its stores and the staging that follows them must not meet
    (64 fields, ten calls, the same bits each time, every field alike)."""
    import torch
    batch = 64
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": "tf32x3"})
    src = torch.from_numpy(np.tile(spectrum(lmax, lmax, 3), (batch, 1))).cuda()
    fm = [torch.empty(batch, 2 * (lmax + 1) * nlat, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    for k in range(10):
        plan.stage_dev("legSynth", src.data_ptr(), fm[min(k, 1)].data_ptr(), batch)
        device.sync()
        assert torch.equal(fm[min(k, 1)], fm[0]), k
    assert torch.equal(fm[0], fm[0][:1].expand_as(fm[0]))
    plan.destroy()


@pytest.mark.parametrize("batch", [33, 49])
def test_first_call_beside_work_on_the_default_stream(device, parity, batch):
    """A tensor-core plan's first call of a batch clears its new operand images;
    work queued on the default stream must not put that clearing off until
    after the kernels that fill them (the context's stream does not wait for
    the default one)."""
    import torch
    lmax, nlat, nphi = 319, 640, 1536
    plan = ShtPlan.create(device, ShtConfig(lmax, lmax, nlat, nphi), {"precision": "tf32x3"})
    ref = O.ShtReference(lmax, lmax, nlat, nphi)
    q = spectrum(lmax, lmax, batch)
    want = ref.synth(q.astype(np.float64))
    src = torch.from_numpy(np.tile(q, (batch, 1))).cuda()
    grid = torch.from_numpy(np.tile(want.astype(np.float32), (batch, 1))).cuda()
    out = [torch.empty_like(grid), torch.empty_like(src)]
    for call, x, y in ((plan.synth_dev, src, out[0]), (plan.analys_dev, grid, out[1])):
        torch.cuda.synchronize()
        torch.cuda._sleep(100_000_000)  # some 50 ms on the default stream
        call(x.data_ptr(), y.data_ptr(), batch)
        torch.cuda.synchronize()
    parity(f"tf32x3 lmax319 B{batch} first synth", O.rel_l2(out[0][-1].cpu().numpy(), want), TOL)
    parity(f"tf32x3 lmax319 B{batch} first analys",
           O.rel_l2(out[1][-1].cpu().numpy(), ref.analys(want.astype(np.float32).astype(np.float64))), TOL)
    plan.destroy()
