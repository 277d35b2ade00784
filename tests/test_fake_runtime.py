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


def test_map_and_count_after_clean_up_and_reset(fake):
    """The original's pair: its callers clean up (the original resets the device there) and count on."""
    fake(r"""
import threading
m = _lib.BinMapF64()
lib.setBinMapF64(C.byref(m), b">", 0.0)
table = (_lib.ConstFieldPtr * 4)()
table[0].p = data.ctypes.data
fi = _lib.BMFieldInfo()
fi.fieldTableMask, fi.elemID, fi.profID = 1, M.ENC_F32, 0
defs = (C.c_int * 3)(64, 40, 40)
fi.pD = defs
fi.pFieldDevPtrTable = table

def pair(where, own=None):
    org, ki, host = _lib.BMOrg(), _lib.KernInfo(), np.zeros(256, np.uint64)
    p = lib.binMapCUDA(C.byref(ki), own, C.byref(org), C.byref(fi), C.byref(m))
    assert p, (where, "map")
    assert ki.dtms[0] == 0.25, (where, ki.dtms[0])
    assert lib.mkfCUDAGetBPFD(C.byref(ki), data.ctypes.data, C.byref(org), p, 0), (where, "count")
    assert lib.mkfCUDAGetBPFDH(C.byref(ki), host.ctypes.data, C.byref(org), p, 0), (where, "count to host")
    assert ki.dtms[1] == 0.25, (where, ki.dtms[1])
    names = [l[1] for l in launches()]
    assert sum("countMap" in n for n in names) == 2, (where, names)

def clean():
    lib.mkfCUDACleanup(1)
    lib.binMapCUDACleanup()

pair("first")
pair("second")
clean()
pair("after clean-up")
clean()
assert fake.cudaDeviceReset() == 0
pair("after clean-up and reset")
assert fake.cudaSetDevice(1) == 0
clean()
pair("second device")
clean()
assert fake.cudaSetDevice(0) == 0
clean()
assert fake.cudaDeviceReset() == 0
t = threading.Thread(target=lambda: pair("thread"))
t.start()
t.join()
assert fake.fake_calls(b"dead event") == 0
# a caller's own buffers and no clean-up: the count needs nothing that a reset takes
org, ki = _lib.BMOrg(), _lib.KernInfo()
own = np.zeros(1 << 16, np.uint32)
assert lib.binMapCUDA(C.byref(ki), own.ctypes.data, C.byref(org), C.byref(fi), C.byref(m))
assert fake.cudaDeviceReset() == 0
assert lib.binMapCUDA(C.byref(ki), own.ctypes.data, C.byref(org), C.byref(fi), C.byref(m))
assert lib.mkfCUDAGetBPFD(C.byref(ki), data.ctypes.data, C.byref(org), own.ctypes.data, 0)
for i in range(40):
    assert lib.mkfCUDAGetBPFD(C.byref(ki), data.ctypes.data, C.byref(org), own.ctypes.data, 0)
    assert fake.cudaDeviceReset() == 0
for i in range(10):
    assert lib.mkfCUDAGetBPFD(C.byref(ki), data.ctypes.data, C.byref(org), own.ctypes.data, 0)
assert fake.fake_events_alive() <= 2
assert fake.fake_calls(b"dead event") == 0
clean()
assert fake.fake_events_alive() == 0, fake.fake_events_alive()
""")


def test_a_tuned_depth_belongs_to_one_kernel(fake):
    """Fields of one size class that different kernels or ways of copying count: a depth and variant
    recorded for one leaves the others alone."""
    fake(r"""
def desc(dt, shape, kind):
    Z, Y, X = shape
    if kind == "aligned":
        return field(shape, dt)
    if kind == "odd":
        return field(shape, dt, 1, (Y * (X + 1), X + 1, 1))
    return field(shape, dt, 0, (2 * Y * X, 2 * X, 2))

def query(d, th):
    dep, var = C.c_int(-1), C.c_int(-1)
    assert lib.mkfTuneQuery(C.byref(d), C.byref(th.ts), C.byref(dep), C.byref(var), None) == 0
    return dep.value, var.value

for dt in (np.float32, np.float64):
    # (nothing reads the fields here, so they may be larger than the memory behind them)
    for shape, ks in (((40, 40, 64), (1, 2, 3, 6, 12, 16)), ((260, 260, 272), (2, 3, 4, 5, 8)), ((520, 520, 544), (1, 2, 5))):
        for k in ks:
            sets = {"spread": M._Thresholds(list(np.linspace(-1.0, 1.0, k)), 4)}
            if 2 < k <= 4 or 4 < k <= 16:
                sets["shared"] = M._Thresholds([100.0 + 1e-3 * i if i < 3 else 200.0 * i for i in range(k)], 4)
            kinds = {}  # what launches -> the descriptions that launch it
            for kind in ("aligned", "odd", "strided"):
                for tn, th in sets.items():
                    d = desc(dt, shape, kind)
                    out = np.zeros((k, 256), np.uint64)
                    launches()
                    assert lib.mkfFieldBPFD(out.ctypes.data, C.byref(d), C.byref(th.ts), 0, None) == 0
                    name = launches()[-1][1]
                    name = name.split("BPFD")[0]
                    if "ballot" in name or name.endswith("thermo"):  # read any field alike
                        kinds.setdefault((name, "", ""), []).append((d, th))
                    else:  # (a threshold set sharing buckets has no variants to choose from)
                        kinds.setdefault((name, kind, tn if "thermoTma" in name and kind == "aligned" else ""), []).append((d, th))
            for me, mine in kinds.items():
                d, th = mine[0]
                variant = 3 if "thermoTma" in me[0] and me[1] == "aligned" and me[2] == "spread" else 0
                assert lib.mkfTuneSet(C.byref(d), C.byref(th.ts), 24, 3, None) == 0
                assert query(d, th) == (24, variant), (me, query(d, th))
                for other, theirs in kinds.items():
                    if other != me:
                        for d2, th2 in theirs:
                            assert query(d2, th2) == (0, 0), (shape, k, me, other)
                assert lib.mkfTuneSet(C.byref(d), C.byref(th.ts), 0, 0, None) == 0
                assert query(d, th) == (0, 0)
""")


def test_a_tuned_depth_gets_its_own_strips(fake):
    """The word kernel's strips for a recorded depth are those that suit it: by the cost that words.cu
    chooses strips by, none is worse than strips of one tile."""
    fake(r"""
def grid(d, th):
    out = np.zeros((th.n, 256), np.uint64)
    assert lib.mkfFieldBPFD(out.ctypes.data, C.byref(d), C.byref(th.ts), 0, None) == 0
    name, smem, blocks, threads = launches()[-1][1:5]
    assert "wordBPFD" in name
    return int(smem), int(blocks), int(threads) // 32

th = M._Thresholds([-0.5, 0.0, 0.5], [4, 1, 2])
for shape in ((64, 512, 1024), (128, 256, 512), (33, 700, 2048)):
    d = field(shape, np.float32)
    for depth in (4, 16, 64, 128):
        assert lib.mkfTuneSet(C.byref(d), C.byref(th.ts), depth, 0, None) == 0
        smem, blocks, warps = grid(d, th)
        W = (smem // warps - 2 * 32 * 144 - 9 * 288) // 128  # state words: 3 (2 W + 3)
        W = (W // 3 - 3) // 2
        tiles, rows, slabs = -(-(shape[2] - 1) // 32), -(-(shape[1] - 1) // 31), -(-(shape[0] - 1) // depth)

        burst = 0.7 / 3 if 128 * tiles * shape[1] * shape[0] > 32e6 else 0.0

        def cost(W, warps):
            rounds = -(-(-(-tiles // W) * rows * slabs) // (148 * warps))
            return rounds * ((depth + 1) * W + 1) * (1 + burst / W) * (warps / 16) ** 0.5

        assert cost(W, warps) <= 1.0001 * cost(1, 16), (shape, depth, W)
        assert lib.mkfTuneSet(C.byref(d), C.byref(th.ts), 0, 0, None) == 0
""")


def test_kernel_of_a_call(fake):
    """Which kernel counts a field, on both sides of each line of the routing."""
    fake(r"""
def kernel(dt, shape, kind, k, m=4):
    Z, Y, X = shape
    d = {"aligned": lambda: field(shape, dt, 0, (Y * (X + 3) // 4 * 4 * 1, (X + 3) // 4 * 4, 1)), "odd": lambda: field(shape, dt, 1, (Y * (X | 1), X | 1, 1)),
         "strided": lambda: field(shape, dt, 0, (2 * Y * X, 2 * X, 2))}[kind]()
    if kind == "aligned":
        d = field(shape, dt, 0, (Y * ((X + 3) // 4 * 4), (X + 3) // 4 * 4, 1))
    rc, names = count(d, k, m)
    assert rc == 0
    n = names[-1]
    return "vote" if "ballot" in n else "word" if "wordBPFD" in n else "staged" if "thermoTma" in n else "global"

F, D = np.float32, np.float64
table = [
    # one threshold
    (F, (64, 127, 128), "aligned", 1, "word"), (F, (64, 129, 128), "aligned", 1, "vote"), (F, (128, 725, 728), "aligned", 1, "word"),
    (F, (128, 725, 728), "odd", 1, "word"), (F, (20, 2000, 2000), "odd", 1, "vote"), (F, (600, 600, 600), "odd", 1, "vote"), (F, (128, 725, 728), "strided", 1, "vote"), (D, (512, 512, 512), "aligned", 1, "vote"),
    # thick fields
    (F, (300, 300, 300), "aligned", 4, "word"), (F, (300, 300, 300), "odd", 3, "word"), (F, (300, 300, 300), "odd", 4, "word"), (F, (200, 200, 200), "odd", 4, "word"),
    (F, (500, 500, 500), "odd", 4, "word"), (F, (600, 600, 600), "odd", 3, "vote"), (F, (600, 600, 600), "odd", 5, "vote"),
    (D, (300, 300, 300), "aligned", 3, "word"), (D, (300, 300, 300), "aligned", 4, "vote"), (D, (200, 200, 200), "aligned", 4, "word"),
    (D, (200, 200, 200), "odd", 2, "vote"), (D, (200, 200, 200), "odd", 3, "word"), (D, (300, 300, 300), "odd", 3, "vote"),
    # strided, flat, narrow
    (F, (200, 200, 200), "strided", 3, "word"), (F, (250, 250, 250), "strided", 3, "vote"), (D, (160, 160, 160), "strided", 3, "word"),
    (D, (200, 200, 200), "strided", 3, "vote"), (D, (200, 200, 200), "strided", 5, "staged"), (D, (300, 300, 300), "strided", 5, "vote"),
    (F, (300, 300, 300), "strided", 5, "staged"), (F, (400, 400, 400), "strided", 5, "vote"), (F, (9000, 9, 1024), "strided", 5, "staged"),
    (D, (300, 300, 300), "strided", 6, "vote"), (D, (200, 200, 200), "strided", 6, "staged"), (F, (300, 300, 300), "strided", 6, "staged"),
    (D, (300, 300, 300), "strided", 8, "global"), (D, (256, 256, 256), "strided", 8, "staged"), (F, (300, 300, 300), "strided", 8, "staged"),
    (F, (2, 2048, 2048), "odd", 2, "vote"), (F, (40, 512, 512), "odd", 2, "word"), (D, (9, 1024, 1024), "aligned", 2, "vote"), (D, (17, 1024, 1024), "aligned", 2, "word"),
    (D, (2, 2048, 2048), "aligned", 5, "vote"), (D, (9, 2048, 2048), "aligned", 5, "staged"), (D, (2, 2048, 2048), "odd", 6, "vote"),
    (F, (512, 6, 1024), "aligned", 2, "vote"), (F, (512, 10, 1024), "aligned", 2, "word"), (F, (512, 10, 1024), "odd", 2, "vote"),
    (F, (17, 512, 512), "odd", 2, "word"), (F, (17, 1024, 1024), "odd", 2, "vote"), (D, (5, 1024, 1024), "aligned", 3, "word"),
    (D, (2000, 1000, 17), "aligned", 3, "word"), (D, (2000, 1000, 20), "aligned", 3, "vote"), (F, (512, 512, 33), "odd", 2, "word"), (F, (512, 512, 40), "odd", 2, "vote"),
    (D, (2000, 20, 1000), "aligned", 4, "word"), (D, (512, 40, 512), "aligned", 4, "vote"), (D, (512, 512, 17), "aligned", 6, "word"),
    (F, (512, 512, 20), "odd", 5, "vote"), (D, (512, 512, 20), "aligned", 6, "vote"), (D, (512, 6, 512), "aligned", 5, "global"), (F, (512, 512, 20), "aligned", 6, "global"), (F, (64, 64, 20), "aligned", 5, "word"),
    (D, (64, 6, 64), "aligned", 6, "word"),
]
for dt, shape, kind, k, want in table:
    assert kernel(dt, shape, kind, k) == want, (dt, shape, kind, k, want, kernel(dt, shape, kind, k))
# thresholds that share a bucket of the rank table
for shape, k, want in (((200, 200, 200), 32, "wordBPFD"), ((210, 210, 210), 23, "wordBPFD"), ((210, 210, 210), 24, "thermoBPFD"), ((210, 210, 210), 8, "wordBPFD")):
    rc, names = count(field(shape, D), k, 4, [300.0 + 0.05 * i for i in range(k)])
    assert rc == 0 and all(want in n for n in names), (shape, k, names)
# differing tests: two by votes, three by words
assert kernel(D, (300, 300, 300), "odd", 2, [4, 1]) == "vote" and kernel(D, (300, 300, 300), "odd", 3, [4, 1, 4]) == "word"
assert kernel(D, (300, 300, 300), "odd", 3, [4, 3, 4]) == "vote"  # (<= is > counted negated)
""")


def test_kernel_of_a_batch(fake):
    """The batched rank table takes a batch none of whose fields needs the word kernel, if it is the faster
    one for its sizes and thresholds; any other batch of up to 8 thresholds is one word kernel launch."""
    fake(r"""
def batch(dt, shapes, ks, plan, masks=None):
    sets = [M._Thresholds(list(np.linspace(-1, 1, k)), 4 if masks is None else masks[i]) for i, k in enumerate(ks)]
    n = len(sets)
    descs = (_lib.MKFFieldDesc * n)(*[field(s, dt) for s in shapes])
    ts = (_lib.MKFThreshSet * n)(*[s.ts for s in sets])
    out = np.zeros((sum(ks), 256), np.uint64)
    launches()
    if plan:
        h = C.c_void_p()
        assert lib.mkfBatchPlanCreate(C.byref(h), out.ctypes.data, descs, ts, n) == 0
        launches()
        assert lib.mkfBatchPlanLaunch(h, None) == 0
        names = [l[1] for l in launches()]
        assert lib.mkfBatchPlanDestroy(h) == 0
    else:
        assert lib.mkfBatchBPFD(out.ctypes.data, descs, ts, n, 0, None) == 0
        names = [l[1] for l in launches()]
    assert all("wordBatch" in x or "thermoBatch" in x for x in names), names
    return "".join(sorted({"w" if "wordBatch" in x else "r" for x in names}))

F, D = np.float32, np.float64
S = lambda n: [(n, n, n)] * 4
for dt, n, k, plan, want in ((F, 16, 3, True, "r"), (F, 60, 8, True, "r"), (F, 90, 4, True, "w"), (F, 90, 5, True, "r"), (F, 150, 3, True, "w"), (F, 150, 8, True, "r"),
                             (D, 90, 3, True, "r"), (D, 110, 3, True, "w"), (D, 110, 4, True, "r"), (F, 16, 8, False, "w"), (F, 90, 8, False, "w"),
                             (F, 110, 5, False, "w"), (F, 110, 6, False, "r"), (D, 110, 8, False, "r"), (F, 16, 2, True, "w"), (F, 16, 12, False, "r")):
    assert batch(dt, S(n), [k] * 4, plan) == want, (dt, n, k, plan)
for plan in (True, False):
    assert batch(F, S(150), [8, 8, 8, 1], plan) == "w" and batch(F, S(150), [8, 8, 8, 3], plan, [4, 4, 4, [4, 1, 2]]) == "w"
    assert batch(F, S(150), [8, 8, 8, 12], plan) == "r" and batch(F, S(150), [1, 8, 8, 12], plan) == "rw"
""")


def test_chunks_of_a_batch(fake):
    """The chunks of a word kernel batch cover every item once, and each is a whole number of rounds of the
    warps that count it, but for the last of a field."""
    fake(r"""
class Args(C.Structure):
    _fields_ = [("tasks", C.c_void_p), ("chunks", C.c_void_p), ("n", C.c_int), ("counter", C.c_void_p)]
class Chunk(C.Structure):
    _fields_ = [("field", C.c_int), ("pad", C.c_int), ("begin", C.c_longlong), ("end", C.c_longlong)]

fake.fake_batch_args.restype = C.POINTER(Args)
for dt, nr in ((np.float32, 4), (np.float64, 2)):
    for strides in (None, (2 * 90 * 90, 2 * 90, 2)):
        for k in (1, 2, 5, 8):
            masks = [4, 1] * k
            sets = [M._Thresholds(list(np.linspace(-1, 1, k)), masks[:k]) for _ in range(40)]
            descs = (_lib.MKFFieldDesc * 40)(*[field((90 - i, 90, 90), dt, 0, strides) for i in range(40)])
            ts = (_lib.MKFThreshSet * 40)(*[s.ts for s in sets])
            out = np.zeros((40 * k, 256), np.uint64)
            h = C.c_void_p()
            lib.mkfSetTuning(0)
            assert lib.mkfBatchPlanCreate(C.byref(h), out.ctypes.data, descs, ts, 40) == 0
            assert lib.mkfBatchPlanLaunch(h, None) == 0
            assert any("wordBatch" in l[1] for l in launches())
            a = fake.fake_batch_args().contents
            chunks = list((Chunk * a.n).from_address(a.chunks))
            mis = strides is None
            W = 2 if k <= 4 else 1
            warp = 2 * 32 * (176 if mis else 144) + 9 * 288 + k * (W * (nr // 2) + 3) * 128
            warps = min(16, (232448 - 1024 * 9 - 2048) // warp)
            for f in range(40):
                mine = sorted((c.begin, c.end) for c in chunks if c.field == f)
                assert mine[0][0] == 0 and all(p[1] == q[0] for p, q in zip(mine, mine[1:])), mine
                assert all((e - b) % warps == 0 for b, e in mine[:-1]) and mine[-1][1] > mine[-1][0], (dt, k, warps, mine)
            assert max(c.end - c.begin for c in chunks) > 0
            assert lib.mkfBatchPlanDestroy(h) == 0
""")


def test_measures_on_other_devices_and_after_a_reset(fake):
    """The measures' tables need no upload, which a reset would undo and a capture would not allow."""
    fake(r"""
r, h = np.zeros((3, 4)), np.ones((3, 256), np.uint64)
for step in (lambda: 0, fake.cudaDeviceReset, lambda: fake.cudaSetDevice(1)):
    assert step() == 0
    launches()
    assert lib.mkfMeasuresF64Dev(r.ctypes.data, h.ctypes.data, 3, None) == 0
    assert ["measuresKernel" in l[1] for l in launches()] == [True]
assert fake.fake_calls(b"cudaMemcpyToSymbol") == 0
""")
