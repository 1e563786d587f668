"""Finalizers in the order of a garbage-collected cycle (a script's globals at
exit): a plan or model whose device has gone is not passed to the library."""
import pytest

from turing_sphere_b200 import GpuModel, ShtPlan, _lib
from turing_sphere_b200.sht import Device


class FakeLibrary:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda handle: self.calls.append(name)


@pytest.mark.parametrize("order,want", [
    ("gpd", ["ts_model_destroy", "ts_sht_plan_destroy", "ts_ctx_destroy"]),
    ("dpg", ["ts_ctx_destroy"]),
    ("pgd", ["ts_sht_plan_destroy", "ts_model_destroy", "ts_ctx_destroy"]),
    ("dgp", ["ts_ctx_destroy"]),
])
def test_finalizers_in_any_order(monkeypatch, order, want):
    lib = FakeLibrary()
    monkeypatch.setattr(_lib, "lib", lambda: lib)
    made = {"d": Device.__new__(Device), "p": ShtPlan.__new__(ShtPlan), "g": GpuModel.__new__(GpuModel)}
    made["d"].handle = made["p"].handle = made["g"].handle = 1
    made["p"].device = made["g"].device = made["d"]
    made["g"].sht = made["p"]
    for key in order:
        made[key].__del__()
    assert lib.calls == want
    for x in made.values():
        x.handle = None
