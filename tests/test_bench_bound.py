"""The bench line names what bounds the products class: its single-vector
products HBM, the starts' products with several vectors the FP64 pipe."""
import importlib
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_products_class_is_not_called_hbm_bound(monkeypatch):
    monkeypatch.syspath_prepend(ROOT)
    b = importlib.import_module("bench")
    monkeypatch.setattr(b, "_peaks", lambda: ({"hbm_gbs": 6400.0, "bf16_tflops_sustained": 1400.0}, "measured"))
    monkeypatch.setattr(b, "_traffic", lambda: {})
    classes = {"residual": dict(launches=10, ms=20.0, work=6.4e10), "trsv": dict(launches=1, ms=1.0, work=3.2e9)}
    r = b.roofline(classes)
    assert r["kernel"] == "residual" and "fp64" in r["bound"] and "hbm" in r["bound"]
    assert r["achieved"] == 3200.0 and r["frac"] == 0.5   # 6.4e9 bytes of Z per launch in 2 ms
    assert b.roofline(classes, "trsv")["bound"] == "hbm"
