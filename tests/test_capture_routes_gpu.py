"""A call on a tensor-core plan can be captured after any call whose operand
images have its size, whichever of the two Legendre routes either takes: the
products' calls size the images that the contraction of up to 64 fields
needs, and a capture for which the products' own scratch is too small takes
the contraction.  Replays against the oracle (1e-5, the transforms' bound)."""
import numpy as np
import pytest

from oracle import oracle as O
from turing_sphere_b200 import ShtConfig, ShtPlan

from .test_leg_gemm_gpu import spectrum

pytestmark = pytest.mark.gpu

LMAX, NLAT, NPHI = 127, 192, 384  # products: synthesis up to 48 fields, analysis up to 16


@pytest.mark.parametrize("call,warm,batch", [("analys", 4, 16), ("analys", 16, 17), ("analys", 4, 64),
                                             ("legAnalys", 4, 16), ("legAnalys", 4, 40),
                                             ("legSynth", 4, 48), ("legSynth", 4, 64)])
def test_capture_after_a_smaller_batch(device, parity, call, warm, batch):
    import torch
    plan = ShtPlan.create(device, ShtConfig(LMAX, LMAX, NLAT, NPHI), {"precision": "tf32x3"})
    ref = O.ShtReference(LMAX, LMAX, NLAT, NPHI)
    q = spectrum(LMAX, LMAX, 3)
    grid = ref.synth(q.astype(np.float64)).astype(np.float32)
    spec = torch.from_numpy(np.tile(q, (64, 1))).cuda()
    spat = torch.from_numpy(np.tile(grid, (64, 1))).cuda()
    fm = torch.zeros(64, (LMAX + 1) * NLAT * 2, device="cuda")
    out = torch.zeros_like(spec)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()

    def run(n):
        at = stream.cuda_stream
        if call == "analys":
            plan.analys_dev(spat.data_ptr(), out.data_ptr(), n, at)
        elif call == "legAnalys":
            plan.stage_dev("legAnalys", fm.data_ptr(), out.data_ptr(), n, at)
        else:
            plan.stage_dev("legSynth", spec.data_ptr(), fm.data_ptr(), n, at)

    if call == "legAnalys":
        plan.stage_dev("fourAnalys", spat.data_ptr(), fm.data_ptr(), 64)
    torch.cuda.synchronize()
    run(warm)
    torch.cuda.synchronize()
    out.zero_()
    if call == "legSynth":
        fm.zero_()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        run(batch)
    graph.replay()
    torch.cuda.synchronize()
    plan.status()
    if call == "legSynth":
        plan.stage_dev("fourSynth", fm.data_ptr(), spat.data_ptr(), batch)
        device.sync()
        got, want = spat, ref.synth(q.astype(np.float64))
    else:
        got, want = out, ref.analys(grid.astype(np.float64))
    for f in (0, batch - 1):
        parity(f"captured {call} of {batch} after {warm}: field {f}", O.rel_l2(got[f].cpu().numpy(), want), 1e-5)
    plan.destroy()


def test_captured_analysis_outlives_a_larger_call(device, parity):
    """A captured analysis of 4 fields replays after a call of 16 and one of
    64 on the same plan: the scratch it holds does not move for them."""
    import torch
    plan = ShtPlan.create(device, ShtConfig(LMAX, LMAX, NLAT, NPHI), {"precision": "tf32x3"})
    ref = O.ShtReference(LMAX, LMAX, NLAT, NPHI)
    q = spectrum(LMAX, LMAX, 5)
    grid = ref.synth(q.astype(np.float64)).astype(np.float32)
    spat = torch.from_numpy(np.tile(grid, (64, 1))).cuda()
    out = torch.zeros(64, q.size, device="cuda")
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    plan.analys_dev(spat.data_ptr(), out.data_ptr(), 4, stream.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        plan.analys_dev(spat.data_ptr(), out.data_ptr(), 4, stream.cuda_stream)
    free = torch.cuda.mem_get_info()[0]
    for batch in (16, 64):
        plan.analys_dev(spat.data_ptr(), out.data_ptr(), batch, stream.cuda_stream)
        torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free  # nothing was allocated or moved
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    want = ref.analys(grid.astype(np.float64))
    for f in (0, 3):
        parity(f"captured analys of 4 after 16 and 64: field {f}", O.rel_l2(out[f].cpu().numpy(), want), 1e-5)
    plan.destroy()
