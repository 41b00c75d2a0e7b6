"""The device-resident step in a context that may use only part of the GPU's
SMs (a green context of sixteen): the tree's cooperative kernel takes fewer
CTAs, and the state is that of the whole GPU bit for bit.  The steps run in
processes of their own, as the context is current for all that they do."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

SCRIPT = """
import ctypes, sys
sys.path.insert(0, {root!r})
sms, out = int(sys.argv[1]), sys.argv[2]
if sms:
    cu = ctypes.CDLL("libcuda.so.1")
    def check(what):
        if what != 0:
            print("no green context:", what)
            sys.exit(77)
    dev, n = ctypes.c_int(), ctypes.c_uint(1)
    res, part, rest = ((ctypes.c_ubyte * 512)() for _ in range(3))  # CUdevResource, 144 bytes
    desc, green, ctx = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    check(cu.cuInit(0))
    check(cu.cuDeviceGet(ctypes.byref(dev), 0))
    check(cu.cuDeviceGetDevResource(dev, res, 1))  # the SMs
    check(cu.cuDevSmResourceSplitByCount(part, ctypes.byref(n), res, rest, 0, sms))
    check(cu.cuDevResourceGenerateDesc(ctypes.byref(desc), part, 1))
    check(cu.cuGreenCtxCreate(ctypes.byref(green), desc, dev, 1))
    check(cu.cuCtxFromGreenCtx(ctypes.byref(ctx), green))
    check(cu.cuCtxSetCurrent(ctx))
import numpy as np
from petar_gb300 import ics, nbody
cl = ics.make_king_cluster(3, 20000, 0.008, W0=6.0, theta=0.4)
with nbody.DeviceNBody(cl) as h:
    h.run(2, 1.0 / 4096)
    s = h.state()
np.savez(out, **s)
"""


def test_step_on_part_of_the_sms(tmp_path):
    states = []
    for sms in (0, 16):
        out = tmp_path / f"state{sms}.npz"
        r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=str(ROOT)), str(sms), str(out)],
                           capture_output=True, text=True, timeout=300)
        if r.returncode == 77:
            pytest.skip(r.stdout)
        assert r.returncode == 0, r.stdout + r.stderr
        states.append(dict(np.load(out)))
    for k in states[0]:
        np.testing.assert_array_equal(states[1][k], states[0][k], err_msg=k)
