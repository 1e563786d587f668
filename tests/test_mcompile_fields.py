"""A model may analyse more fields per instance than a tile of the FP32
products holds (8 to 32): it compiles without them, or is refused where the
tensor-core path has too many outputs, and the host code does not divide by
the zero instances that such a tile would take."""
import ctypes as C

import pytest

from turing_sphere_b200 import _lib


def source(n):
    terms = [f"analys(u.^{2 + k % 5} * {k + 1})" for k in range(n)]
    return ("function [U, u] = init(noise)\n  U = analys(noise);\n  u = synth(U);\nend\n"
            "function [Un, u] = step(U, lam, c, dt)\n  u = synth(U);\n"
            f"  Un = (U + dt * ({' + '.join(terms)})) ./ (1 + c * lam);\nend\n")


@pytest.mark.parametrize("precision,n,accepted",
                         [(_lib.TS_PREC_FP32, n, True) for n in (8, 9, 32, 33, 40)] +
                         [(_lib.TS_PREC_TF32X3, n, n <= 16) for n in (8, 9, 17, 32, 33, 40)])
def test_analysed_fields_per_instance(precision, n, accepted):
    buf, k, launches, err = C.create_string_buffer(1 << 16), C.c_int(), C.c_int(), _lib.CompileError()
    rc = _lib.lib().ts_model_check(63, 63, 96, 192, source(n).encode(), _lib.cstr_array(["U"]), 1,
                                   _lib.cstr_array(["u"]), 1, _lib.cstr_array(["c", "dt"]), 2, 1, precision,
                                   buf, len(buf), C.byref(k), C.byref(launches), C.byref(err))
    if not accepted:
        assert rc == _lib.TS_ERR_COMPILE and b"too many" in err.message
        return
    assert rc == _lib.TS_OK, err.message.decode()
    assert f"{n} analys" in buf.value.decode()
