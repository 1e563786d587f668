"""The fused phase's registers are held down only where a second CTA can use
them: at nphi 2048 (two species, 8 rows: 147 KB of shared memory) the kernel
spills nothing.  Compiles the generated step of a model for that shape."""
import ctypes as C
import os
import re
import shutil
import subprocess

import pytest

from turing_sphere_b200 import _lib, mModelByKey

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
KERNELS = os.path.join(os.path.dirname(_lib.__file__), "csrc", "kernels")


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_phase_of_two_species_at_nphi_2048_spills_nothing(tmp_path):
    model = mModelByKey("schnakenberg")
    buf, k, n, err = C.create_string_buffer(1 << 18), C.c_int(), C.c_int(), _lib.CompileError()
    params = [p.key for p in model.params]
    rc = _lib.lib().ts_model_check(341, 341, 1024, 2048, model.source.encode(), _lib.cstr_array(model.state), 2,
                                   _lib.cstr_array(model.species), 2, _lib.cstr_array(params), len(params), 64,
                                   _lib.TS_PREC_TF32X3 | _lib.TS_CHECK_SOURCE, buf, len(buf), C.byref(k),
                                   C.byref(n), C.byref(err))
    assert rc == _lib.TS_OK, err.message.decode()
    prog = re.search(r"struct TsProg_s0 \{.*?\n\};\n", buf.value.decode(), re.S).group(0)
    src = tmp_path / "phase.cu"
    src.write_text('#include "ts_common.cuh"\n#include "fft2.cuh"\n' + prog +
                   "template __global__ void ts_f2_phase<TsProg_s0, 32, 32, 8, true>(TsFftTab, TsPhaseIO);\n")
    out = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                          "--expt-relaxed-constexpr", "-Xptxas", "-v", "-I", KERNELS, "-c", str(src), "-o",
                          str(tmp_path / "phase.o")], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    spills = re.findall(r"(\d+) bytes spill stores", out.stderr)
    assert spills and all(int(s) == 0 for s in spills), out.stderr
