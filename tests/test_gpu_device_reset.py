"""The device-pointer diffusion around a reset of the device by the application.

The library keeps a memory pool per device, and a reset ends it with everything else
in the context: a call after the reset may report an error but may not touch the old
pool (its handle dangles, which is why this runs in a process of its own).
"""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import sys
import numpy as np
import marl_cuda as marl
from cuda.bindings import driver as cu


def ok(r):
    assert r[0] == cu.CUresult.CUDA_SUCCESS, r
    return r[1] if len(r) == 2 else None


ok(cu.cuInit(0))
dev = ok(cu.cuDeviceGet(0))
p = marl.default_params()
field = np.random.default_rng(0).random((13, 21, 37, 12), dtype=np.float32)
occ = np.zeros((13, 21, 37), np.uint8)


def call():
    ok(cu.cuCtxSetCurrent(ok(cu.cuDevicePrimaryCtxRetain(dev))))
    f, s, o = ok(cu.cuMemAlloc(field.nbytes)), ok(cu.cuMemAlloc(field.nbytes)), ok(cu.cuMemAlloc(occ.nbytes))
    ok(cu.cuMemcpyHtoD(f, field.ctypes.data, field.nbytes))
    ok(cu.cuMemcpyHtoD(o, occ.ctypes.data, occ.nbytes))
    try:
        for _ in range(3):
            marl.diffuse_device(int(f), int(s), int(o), (37, 21, 13), p, SUBSTEPS)
    except marl.MarlError as e:
        return e.status_name
    return "OK"


first = call()
assert first == "OK", first
for _ in range(2):
    ok(cu.cuDevicePrimaryCtxReset(dev))
    got = call()
    assert got in ("OK", "CUDA"), got
print("ENDED WELL")
"""


@pytest.mark.parametrize("substeps", [3, 10])  # by tiles; in one kernel
def test_calls_around_a_reset(marl, substeps):
    pytest.importorskip("cuda.bindings.driver")
    env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "marl-ochre_b200"))
    r = subprocess.run([sys.executable, "-c", CHILD.replace("SUBSTEPS", str(substeps))], env=env, capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0 and "ENDED WELL" in r.stdout, r.stderr[-2000:]
