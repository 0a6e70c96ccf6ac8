"""What a program pays once: the first context of a process (GPU)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FIRST = """
import sys, time
sys.path.insert(0, %r)
import torch
torch.zeros(1, device="cuda")
torch.cuda.synchronize()
from mbx_b200 import capi
capi.lib()
t = time.perf_counter()
capi.Context(0)
print("seconds", time.perf_counter() - t)
""" % ROOT


def test_first_context_of_a_process():
    """The code and coefficients of every evaluator go to the device with the
    first context: about 80 MB, 0.05 s where nothing has to be decompressed
    (0.26 s with compressed images and line tables).  The limit leaves a
    factor of three for a busy host, and one of two processes has to meet it."""
    times = []
    for _ in range(2):
        r = subprocess.run([sys.executable, "-c", FIRST], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr[-2000:]
        times.append(float(r.stdout.split()[-1]))
    assert min(times) < 0.15, times
