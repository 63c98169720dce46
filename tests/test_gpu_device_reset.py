"""The library keeps page-locked records from case to case.  After the host
program has reset its device (in a process of its own, with no case alive),
new cases get records of the new context: as many as there are, read and
stepped like those before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes, sys
import lbm_ddf_b200 as lbm

rt = ctypes.CDLL(sys.argv[1])
p = lbm.make_params(24, 8, 20, rayleigh=1e4, storage="f32")


def read(cases):
    out = []
    for i, c in enumerate(cases):
        c.init_conduction(i, 1e-2)
        c.step(i % 4)
        out.append(c.observables())
    return out


first = None
for _ in range(3):
    cases = [lbm.Case(p) for _ in range(70)]
    got = read(cases)
    assert first is None or got == first
    first = got
    for c in cases[::2] + cases[1::2]:
        c.close()
    with lbm.Case(p) as c:
        assert read([c]) == first[:1]
    assert rt.cudaDeviceReset() == 0
print("fine")
"""


def test_cases_after_a_device_reset(lbm):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from test_gpu_obs_tail_rows import _cudart

    root = os.path.dirname(os.path.dirname(os.path.abspath(lbm.__file__)))
    r = subprocess.run([sys.executable, "-c", PROGRAM, _cudart()._name], cwd=root, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "fine", r.stderr[-2000:]
