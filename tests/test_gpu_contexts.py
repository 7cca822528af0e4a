"""The order in which a C program destroys a context and its handles."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes
from itk_gb300 import _capi
L = _capi.lib()
ctx, metrics, batch = ctypes.c_void_p(), [ctypes.c_void_p() for _ in range(3)], ctypes.c_void_p()
assert L.gb_ctx_create(0, ctypes.byref(ctx)) == 0
for m in metrics:
    assert L.gb_metric_create(ctx, 0, ctypes.byref(m)) == 0
assert L.gb_batch_create(ctx, ctypes.byref(batch)) == 0
assert L.gb_metric_destroy(metrics[0]) == 0
assert L.gb_ctx_destroy(ctx) == 0
assert L.gb_metric_destroy(metrics[1]) == 0
assert L.gb_batch_destroy(batch) == 0
assert L.gb_metric_destroy(metrics[2]) == 0
print("done")
"""


def test_context_destroyed_before_its_handles():
    # freed host memory is filled, so that a use of it does not pass by chance
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, env=dict(os.environ, MALLOC_PERTURB_="165"),
                       capture_output=True, text=True, timeout=30)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr
