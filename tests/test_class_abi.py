"""Compiled callers of the C++ classes: every member function that the public headers declare without a body is a
symbol of the library (an inline one would be missing for callers built before it became inline)."""
import os
import re
import subprocess

from libgwmodel_gb300 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fit_predict_and_diagnostics_are_exported():
    _lib.lib()
    so = os.path.join(ROOT, "libgwmodel_gb300", "libgwgpu.so")
    out = subprocess.run(["nm", "-D", "-C", "--defined-only", so], check=True, capture_output=True, text=True).stdout
    for name in ("gwm::GWRBasic::fit()", "gwm::GWRBasic::fitInPlace()", "gwm::GWRBasic::predict(gwm::mat const&)",
                 "gwm::GWRMultiscale::fit()"):
        assert re.search(r" T " + re.escape(name) + r"$", out, re.M), name
