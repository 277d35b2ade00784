"""Performance cases of the counting paths: what a program that uses this package has it do.

A case is a dict of plain values; `prepare` makes its fields on the GPU (or in pinned host memory)
from a seed, `run` makes one pass through the public entry points and returns the whole output,
`exact` forms the computed numbers again in 64 bits with plain torch. The fields are synthetic:
Gaussian random fields (smooth, many thresholds), sums of plane waves (an in-situ series) and
unions of balls with noise (one threshold near the surface).
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import mkf_b200
from mkf_b200 import _lib

RELATIONS = {"<": 1, "=": 2, "<=": 3, ">": 4, "!=": 5, ">=": 6}

# Symmetry group (a..v = 0..21) of each of the 256 cell patterns, and the groups' weights.
GROUPS = ("abbcbcdfbdcfcffibcdfdfhjeggkgknqbdcfeggkdhfjgnkqcffigknqgnkqlppt"
          "bdegcfgkdhgnfjkqcfgkfinqgnlpkqptdhgngnlphmnonopsfjkqkqptnopspsru"
          "bedgdghncgfkfkjqdghnhnmoglnpnposcgfkglnpfniqkpqtfkjqnposkpqtprsu"
          "cgglfknpfnkpiqqtfknpjqoskpprqtsufnkpkpprjoqsqstuiqqtqtsuqstutuuv")
W_CHI = (0, 3, 0, 6, 6, -3, 3, 9, 0, -6, -6, 0, 12, 0, -3, -8, -3, -12, -6, 0, 3, 0)
W_S = (0, 0.944412, 1.05178, 0.921095, 0.496906, 0.949947, 0.865898, 0.793181, 0.926631, 0.638921, 0.764068,
       0.784616, 0.874463, 0.868666, 0.557639, 0.682786, 0.923863, 0.496906, 0.737983, 0.65947, 0.0812817, 0)
W_M = (0, 0.763019, 0.642656, 0.616236, 0.686801, 0.187756, 0.167269, 0.161335, 0, -0.431447, -0.287632,
       0, 0, -0.143816, -0.592783, -0.540019, -0.475387, -0.686801, -0.616236, -0.727774, -0.331571, 0)


def listed():
    return [
        # the smallest call: one block of a domain decomposition, counted and measured each time
        # step, where launches and latency are the whole cost
        {"name": "field_64_f32_k1", "kind": "field", "content": "ball", "z": 64, "y": 64, "x": 64, "dtype": "f32",
         "k": 1, "rel": ">"},
        # the plain method's workload: one 256^3 image, one threshold, in one fused call
        {"name": "field_256_f32_k1", "kind": "field", "content": "ball", "z": 256, "y": 256, "x": 256,
         "dtype": "f32", "k": 1, "rel": ">"},
        # the same image through the original pair of calls (map, then counts), as a program
        # written for the original library makes them
        {"name": "pair_256_f32", "kind": "pair", "content": "ball", "z": 256, "y": 256, "x": 256, "dtype": "f32",
         "rel": ">"},
        # the benchmark: a large double-precision field, its functionals as curves over 16 thresholds
        {"name": "field_1024_f64_k16", "kind": "field", "content": "grf", "z": 1024, "y": 1024, "x": 1024,
         "dtype": "f64", "k": 16, "rel": ">"},
        # an ordinary single-precision field over 8 thresholds (a served request)
        {"name": "field_512_f32_k8", "kind": "field", "content": "grf", "z": 512, "y": 512, "x": 512, "dtype": "f32",
         "k": 8, "rel": ">="},
        # a cropped scan: odd extents, rows off the 16-byte boundaries, 12 thresholds from below
        {"name": "field_odd_f64_k12", "kind": "field", "content": "grf", "z": 333, "y": 401, "x": 487, "dtype": "f64",
         "k": 12, "rel": "<"},
        # a slab of the in-situ series: wide planes, three thresholds
        {"name": "insitu_f32_k3", "kind": "field", "content": "waves", "z": 256, "y": 2048, "x": 2048, "dtype": "f32",
         "k": 3, "rel": ">"},
        # thresholds of several relations in one read (excursion sets from both sides)
        {"name": "field_mixed_f32_k5", "kind": "field", "content": "grf", "z": 288, "y": 320, "x": 384, "dtype": "f32",
         "k": 5, "rel": "mixed"},
        # counts and descriptive moments from one read
        {"name": "moments_400_f64_k2", "kind": "moments", "content": "grf", "z": 400, "y": 400, "x": 400,
         "dtype": "f64", "k": 2, "rel": ">"},
        # many uneven images in one launch, the plan kept between passes
        {"name": "batch_96_f32_k1", "kind": "batch", "n": 96, "lo": 17, "hi": 400, "shapes": 3, "dtype": "f32",
         "kmax": 1, "rel": ">"},
        # a burst of requests to the request loop: 1-8 thresholds, both element types
        {"name": "serve_64_mixed", "kind": "serve", "n": 64, "lo": 32, "hi": 320, "shapes": 5, "dtype": "both",
         "kmax": 8, "rel": ">"},
        # a field that lies in pinned host memory
        {"name": "host_384_f32_k3", "kind": "host", "content": "grf", "z": 384, "y": 384, "x": 384, "dtype": "f32",
         "k": 3, "rel": ">"},
    ]


def _extents(rng, lo, hi):
    """z, y, x of a volume log-uniform between lo and hi voxels, extents within a factor of 4."""
    vol = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a = [math.exp(rng.uniform(-math.log(2.0), math.log(2.0))) for _ in range(3)]
    g = (a[0] * a[1] * a[2]) ** (1.0 / 3.0)
    return [max(8, int(round(vol ** (1.0 / 3.0) * v / g))) for v in a]


def draw(rng):
    kind = rng.choice(["field"] * 7 + ["pair", "moments", "batch", "serve", "host"])
    dtype = rng.choice(["f32", "f32", "f64"])
    if kind in ("batch", "serve"):
        return {"kind": kind, "n": rng.randint(16, 96), "lo": rng.randint(12, 40), "hi": rng.randint(120, 320),
                "shapes": rng.randrange(1 << 20), "dtype": rng.choice([dtype, "both"]), "kmax": rng.randint(1, 12),
                "rel": rng.choice([">", ">=", "<", "<="])}
    top = {"field": 2 ** 29, "pair": 2 ** 27, "moments": 2 ** 27, "host": 2 ** 26}[kind]
    z, y, x = _extents(rng, 2 ** 15, top)
    if rng.random() < 0.35:
        x = (x + 31) // 32 * 32
    case = {"kind": kind, "content": rng.choice(["grf", "grf", "waves", "ball"]), "z": z, "y": y, "x": x,
            "dtype": dtype, "rel": rng.choice([">", ">", ">=", "<", "<="])}
    if kind == "field":
        case["k"] = min(32, int(math.exp(rng.uniform(0.0, math.log(33.0)))))
        if case["k"] > 1 and rng.random() < 0.2:
            case["rel"] = "mixed"
        if rng.random() < 0.15:
            case["roi"] = True  # an inner region of a larger array
    elif kind in ("moments", "host"):
        case["k"] = rng.randint(1, 2) if kind == "moments" else rng.randint(1, 16)
    return case


# ------------------------------------------------------------------ fields

def _grf(shape, dtype, g, sigma=4.0):
    """White noise, periodic Gaussian smoothing, zero mean and unit variance."""
    w = torch.fft.rfftn(torch.randn(shape, dtype=dtype, device="cuda", generator=g))
    for d, n in enumerate(shape):
        fr = torch.fft.rfftfreq(n, device="cuda", dtype=dtype) if d == 2 else torch.fft.fftfreq(n, device="cuda", dtype=dtype)
        w *= torch.exp(-0.5 * (sigma * 2 * math.pi * fr) ** 2).view([-1 if i == d else 1 for i in range(3)])
    f = torch.fft.irfftn(w, s=shape)
    del w
    f -= f.mean()
    f /= f.std()
    return f.contiguous()


def _waves(shape, dtype, g, n=256):
    """Sum of plane waves, wave numbers 0.05 .. 0.1 per voxel, unit variance."""
    d = torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=g)
    u = torch.rand((n, 2), dtype=torch.float64, device="cuda", generator=g)
    k = d / d.norm(dim=1, keepdim=True) * (0.05 + 0.05 * u[:, :1])
    ax, ay, az = (torch.exp(1j * torch.arange(m, dtype=torch.float64, device="cuda")[:, None] * k[None, :, c]).to(torch.complex64)
                  for c, m in ((0, shape[2]), (1, shape[1]), (2, shape[0])))
    az = az * torch.exp(2j * math.pi * u[:, 1]).to(torch.complex64)
    f = torch.empty(shape, dtype=dtype, device="cuda")
    for z0 in range(0, shape[0], 16):
        p = torch.matmul(ay[None] * az[z0:z0 + 16, None, :], ax.T)
        f[z0:z0 + 16] = p.real * math.sqrt(2.0 / n)
    return f


def _balls(shape, dtype, g, rng):
    """Largest of r - |p - c| over some balls, with noise."""
    f = torch.full(shape, -50.0, dtype=dtype, device="cuda")
    for _ in range(rng.randint(1, 32)):
        c = [rng.random() * n for n in shape]
        r = rng.uniform(2.0, min(40.0, 2.0 + 0.4 * max(shape)))
        lo = [max(0, int(c[i] - r - 1)) for i in range(3)]
        hi = [min(shape[i], int(c[i] + r + 2)) for i in range(3)]
        ax = [(torch.arange(a, b, device="cuda", dtype=dtype) - m) ** 2 for a, b, m in zip(lo, hi, c)]
        box = f[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]]
        torch.maximum(box, r - torch.sqrt(ax[0].view(-1, 1, 1) + ax[1].view(1, -1, 1) + ax[2].view(1, 1, -1)), out=box)
    f += torch.randn(shape, dtype=dtype, device="cuda", generator=g) * 0.1
    return f


def _field(content, shape, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.float32 if dtype == "f32" else torch.float64
    if content == "grf":
        return _grf(shape, dt, g)
    return _waves(shape, dt, g) if content == "waves" else _balls(shape, dt, g, random.Random(seed))


def _thresholds(k, rel, content="grf"):
    """k values over the field's range with their relation masks (one, or one per value)."""
    top = 2.0 if k > 3 else 0.5
    t = [0.0] if k == 1 else np.linspace(-top, top, k).tolist()
    if rel == "mixed":
        return t, [RELATIONS[("<", "<=", "!=", ">", ">=", "=")[i % 6]] for i in range(k)]
    return t, RELATIONS[rel]


def _members(case):
    """(shape, dtype, k) of a batch's or burst's fields."""
    rng = random.Random(case["shapes"])
    got = []
    for _ in range(case["n"]):
        if case["kind"] == "batch":
            shape = [rng.randint(case["lo"], case["hi"]) for _ in range(3)]
        else:
            shape = _extents(rng, case["lo"] ** 3, case["hi"] ** 3)
        dtype = case["dtype"] if case["dtype"] != "both" else ("f32" if rng.random() < 0.7 else "f64")
        got.append((tuple(shape), dtype, rng.randint(1, case["kmax"])))
    return got


# ------------------------------------------------------------------ the cases

class _Pair:
    """The arguments a caller of the original pair builds once."""

    def __init__(self, f, rel):
        z, y, x = f.shape
        self.f = f
        self.defs = (C.c_int * 3)(x, y, z)
        self.table = (_lib.ConstFieldPtr * 4)()
        self.table[0].p = f.data_ptr()
        self.fi = _lib.BMFieldInfo()
        self.fi.fieldTableMask = 1
        self.fi.elemID = _lib.ENC_F32 if f.dtype == torch.float32 else _lib.ENC_F64
        self.fi.pD = self.defs
        self.fi.pFieldDevPtrTable = self.table
        self.bm, self.org, self.ki = _lib.BinMapF64(), _lib.BMOrg(), _lib.KernInfo()
        L = mkf_b200.lib()
        L.setBinMapF64(C.byref(self.bm), rel.encode(), 0.0)
        self.map = torch.zeros(int(L.setBMO(None, self.defs, bytes([0]))), dtype=torch.int32, device=f.device)
        self.counts = np.zeros(256, np.uint64)

    def __call__(self):
        L = mkf_b200.lib()
        if not L.binMapCUDA(C.byref(self.ki), self.map.data_ptr(), C.byref(self.org), C.byref(self.fi), C.byref(self.bm)):
            raise RuntimeError("binMapCUDA")
        if not L.mkfCUDAGetBPFDH(C.byref(self.ki), self.counts.ctypes.data, C.byref(self.org), self.map.data_ptr(), 3):
            raise RuntimeError("mkfCUDAGetBPFDH")
        return self.map, self.counts


def _one(case, seed):
    shape = (case["z"], case["y"], case["x"])
    if case.get("roi"):
        f = _field(case["content"], tuple(n + 6 for n in shape), case["dtype"], seed)
        return f[3:3 + shape[0], 2:2 + shape[1], 1:1 + shape[2]]
    return _field(case["content"], shape, case["dtype"], seed)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("batch", "serve"):
        members = _members(case)
        s["fields"] = [_field("ball", shape, dt, seed * 1000 + i) for i, (shape, dt, _) in enumerate(members)]
        s["t"], s["m"] = zip(*(_thresholds(k, case["rel"]) for _, _, k in members))
        torch.cuda.synchronize()
        if kind == "batch":
            s["plan"] = mkf_b200.BatchPlan(s["fields"], s["t"], s["m"])
        else:
            s["server"] = mkf_b200.Server(hbm_budget=1 << 28)
        return s
    f = _one(case, seed)
    if kind == "pair":
        s["pair"] = _Pair(f, case["rel"])
        torch.cuda.synchronize()
        return s
    s["t"], s["m"] = _thresholds(case["k"], case["rel"])
    if kind == "host":
        h = torch.empty(f.shape, dtype=f.dtype, pin_memory=True)
        h.copy_(f)
        s["pinned"], f = h, h.numpy()
    s["field"] = f
    return s


def run(state):
    kind = state["kind"]
    if kind == "field":
        counts = mkf_b200.field_bpfd(state["field"], state["t"], state["m"])
        return counts, mkf_b200.measures_dev(counts)
    if kind == "moments":
        return mkf_b200.field_bpfd_moments(state["field"], state["t"], state["m"])
    if kind == "pair":
        return state["pair"]()
    if kind == "batch":
        return state["plan"].launch()
    if kind == "serve":
        srv = state["server"]
        tickets = [srv.submit(f, t, m, host_out=True) for f, t, m in zip(state["fields"], state["t"], state["m"])]
        return np.concatenate([srv.wait(tk)[0] for tk in tickets])
    return mkf_b200.field_bpfd_host(state["field"], state["t"], state["m"])


def work(case):
    """Each field read once, each count written once (the map of the pair written and read)."""
    size = {"f32": 4, "f64": 8}
    if case["kind"] in ("batch", "serve"):
        return {"bytes": sum(math.prod(shape) * size[dt] + k * 2048 for shape, dt, k in _members(case)), "flops": 0.0}
    n = case["z"] * case["y"] * case["x"]
    if case["kind"] == "pair":
        return {"bytes": n * size[case["dtype"]] + 2 * (case["z"] * case["y"] * ((case["x"] + 31) // 32) * 4) + 2048, "flops": 0.0}
    return {"bytes": n * size[case["dtype"]] + case["k"] * (2048 + 32), "flops": 0.0}


# ------------------------------------------------------------------ the same numbers in 64 bits

def _maps(f, t, m):
    """The map of f for threshold t and relation mask m."""
    f = f.double()
    return ((f < t) & bool(m & 1)) | ((f == t) & bool(m & 2)) | ((f > t) & bool(m & 4))


def _counts(f, t, m):
    total = torch.zeros(256, dtype=torch.int64, device=f.device)
    step = max(1, (1 << 26) // (f.shape[1] * f.shape[2]))
    for z0 in range(0, f.shape[0] - 1, step):
        b = _maps(f[z0:z0 + step + 1], t, m).to(torch.uint8)
        code = None
        for i in range(8):
            x, y, z = i & 1, (i >> 1) & 1, (i >> 2) & 1
            c = b[z:b.shape[0] - 1 + z, y:b.shape[1] - 1 + y, x:b.shape[2] - 1 + x] * (1 << i)
            code = c if code is None else code + c
        total += torch.bincount(code.reshape(-1).int(), minlength=256)
    return total


def _measures(counts):
    h = counts.double().cpu().numpy()
    group = np.array([ord(c) - ord("a") for c in GROUPS])
    w = np.stack([np.arange(256) & 1, np.array(W_S)[group], np.array(W_M)[group], np.array(W_CHI)[group] / 24.0], 1)
    return h @ w


def exact(case, seed):
    if case["kind"] not in ("field", "moments"):
        return None
    f = _one(case, seed)
    t, m = _thresholds(case["k"], case["rel"])
    m = [m] * len(t) if isinstance(m, int) else m
    if case["kind"] == "field":
        return None, _measures(torch.stack([_counts(f, a, b) for a, b in zip(t, m)]))
    d, got = f.double(), []
    for a, b in zip(t, m):
        on = _maps(f, a, b)
        got.append([[float(d[q].sum()), float(d[q].square().sum())] for q in (~on, on)])
    return None, np.array(got)
