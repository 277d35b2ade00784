"""The library's host side on several devices and across device resets, without a GPU: libMKF.so is
loaded in a child process over a stand-in CUDA runtime (fake_cudart.cpp), which refuses launches and
handles as the real one does and runs no kernel."""
import os
import shutil
import subprocess
import sys

import pytest

from conftest import REPO

CHILD = r"""
import ctypes as C, sys
sys.path.insert(0, %r)
import numpy as np
import mkf_b200 as M
from mkf_b200 import _lib
fake = C.CDLL("libcudart.so.12")
fake.fake_launches.restype = C.c_char_p
lib = M.lib()
data = np.zeros(1 << 20, np.float64)

def launches():
    return [l.split() for l in fake.fake_launches().decode().splitlines()]

def field(shape, dtype=np.float64, off=0, strides=None):
    return M._field_desc(data.ctypes.data + off * np.dtype(dtype).itemsize, M.ENC_F32 if dtype == np.float32 else M.ENC_F64, shape, strides)

def count(d, k, m=4, t=None):
    th = M._Thresholds(list(np.linspace(-1.0, 1.0, k)) if t is None else t, m)
    out = np.zeros((k, 256), np.uint64)
    rc = lib.mkfFieldBPFD(out.ctypes.data, C.byref(d), C.byref(th.ts), 0, None)
    return rc, [l[1] for l in launches()]
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("fake")
    (d / "version").write_text("libcudart.so.12 { global: *; };\n")
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", os.path.join(REPO, "tests", "fake_cudart.cpp"),
                    "-Wl,-soname,libcudart.so.12", f"-Wl,--version-script={d / 'version'}", "-o", str(d / "libcudart.so.12")], check=True)

    def run(body):
        env = dict(os.environ, LD_LIBRARY_PATH=str(d) + ":" + os.environ.get("LD_LIBRARY_PATH", ""))
        r = subprocess.run([sys.executable, "-c", CHILD % REPO + body], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout

    return run


CALLS = r"""
def calls(where):
    for dt in (np.float32, np.float64):
        for off in (0, 1):
            for k in (1, 3, 4, 6, 7, 16, 20, 32):
                rc, names = count(field((40, 40, 64), dt, off), k)
                assert rc == 0 and names, (where, dt, off, k, lib.mkfLastError())
            assert count(field((40, 40, 64), dt, off), 9, [4, 1, 2] * 3)[0] == 0, where
            rc, names = count(field((20, 20, 40), dt, off, (4096, 96, 2)), 8)
            assert rc == 0 and any("thermoTma" in n for n in names), (where, names)
            mom = np.zeros((2, 2, 2))
            out = np.zeros((2, 256), np.uint64)
            th = M._Thresholds([0.0, 0.5], 4)
            d = field((40, 40, 64), dt, off)
            assert lib.mkfFieldBPFDMoments(out.ctypes.data, mom.ctypes.data, C.byref(d), C.byref(th.ts), 0, None) == 0, where
            sets = [M._Thresholds(list(np.linspace(-1, 1, k)), 4) for k in (1, 5, 12, 32)]
            descs = (_lib.MKFFieldDesc * 4)(*[d] * 4)
            ts = (_lib.MKFThreshSet * 4)(*[s.ts for s in sets])
            big = np.zeros((50, 256), np.uint64)
            assert lib.mkfBatchBPFD(big.ctypes.data, descs, ts, 4, 0, None) == 0, (where, lib.mkfLastError())
            names = {l[1] for l in launches()}
            assert any("wordBatch" in n for n in names) and any("thermoBatch" in n for n in names), names
"""


def test_every_kernel_launches_on_a_second_device(fake):
    fake(CALLS + r"""
calls("first device")
assert fake.cudaSetDevice(1) == 0
calls("second device")
assert fake.cudaSetDevice(0) == 0
calls("first device again")
""")


def test_every_kernel_launches_after_a_device_reset(fake):
    fake(CALLS + r"""
calls("before")
assert fake.cudaDeviceReset() == 0
calls("after")
""")
