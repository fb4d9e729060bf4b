"""The checked build takes the paths that only large meshes take (products on the
integer pipe, part-wet lists longer than the lane groups take), the getters' row
kernels and the bed records' kernels without a bad index, with the product build's
bits."""
import json
import os
import subprocess
import sys

import pytest

from swe_fvm_gb300.build import build

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(checked: bool) -> dict:
    env = dict(os.environ, SWE_GB300_CHECKED="1" if checked else "0", PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, os.path.join(ROOT, "tests", "checked_run_large.py")], capture_output=True,
                       text=True, env=env, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_checked_build_on_large_meshes(gpu):
    build(checked=True)
    a, b = _run(False), _run(True)
    assert not a.pop("checked") and b.pop("checked")
    assert a.pop("library") != b.pop("library")
    ga, gb = a.pop("adjoint_grads"), b.pop("adjoint_grads")
    assert a == b
    for x, y in zip(ga, gb):  # (node sums are atomic: their order varies by rounding)
        assert x > 0 and abs(x - y) <= 1e-12 * x
