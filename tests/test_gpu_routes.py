"""Fields on both sides of the lines between the counting kernels, against a plain count of the 256 patterns:
strided, flat and narrow fields, rows off 16-byte boundaries, one test and two, special values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def plain_counts(f, t, m):
    """The 256 pattern counts of a (Z, Y, X) tensor, threshold t, relation mask m (1 <, 2 =, 4 >; NaN is
    "equal", as the original maps it)."""
    import torch

    f = f.double()
    b = (((f < t) & bool(m & 1)) | ((f > t) & bool(m & 4)) | (~(f < t) & ~(f > t) & bool(m & 2))).to(torch.uint8)
    code = None
    for i in range(8):
        x, y, z = i & 1, (i >> 1) & 1, (i >> 2) & 1
        c = b[z:b.shape[0] - 1 + z, y:b.shape[1] - 1 + y, x:b.shape[2] - 1 + x] * (1 << i)
        code = c if code is None else code + c
    return torch.bincount(code.reshape(-1).int(), minlength=256)


def make(shape, dtype, cuda, step=1, off=0):
    """A smooth field with noise and special values; rows `off` elements into a wider array, every `step`-th
    element of a row."""
    import torch

    Z, Y, X = shape
    g = torch.Generator(device=cuda).manual_seed(X)
    big = torch.randn((Z, Y, X * step + off + 1), device=cuda, generator=g, dtype=getattr(torch, dtype)) * 0.3
    big += torch.sin(torch.arange(Y, device=cuda) * 0.1)[None, :, None] + torch.sin(torch.arange(Z, device=cuda) * 0.2)[:, None, None]
    flat = big.view(-1)
    for i, v in enumerate((float("nan"), float("inf"), float("-inf"), -0.0)):
        flat[7 + i::9973] = v
    return big[:, :, off:off + X * step:step]


# below and above 2^21 voxels; Z 2 .. 10, Y 6 .. 63, X 20 .. 64
SHAPES = [(2, 1024, 1023), (2, 1030, 1031), (7, 620, 611), (10, 500, 503), (300, 6, 1201), (400, 20, 301), (160, 63, 257),
          (330, 330, 20), (260, 261, 31), (190, 191, 63), (130, 129, 131), (129, 126, 128)]


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("shape", SHAPES)
def test_counts_by_every_route(mkf, cuda, dtype, shape):
    import torch

    for step, off in ((1, 0), (1, 1), (2, 0)):
        f = make(shape, dtype, cuda, step, off)
        for k, m in ((1, 4), (2, 3), (2, [4, 1]), (2, [2, 6]), (3, 6), (4, 1), (5, 4), (6, 3), (6, [4, 1, 2] * 2), (8, 1)):
            t = np.linspace(-1.0, 1.2, k)
            got = mkf.field_bpfd(f, t, m)
            want = torch.stack([plain_counts(f, v, w) for v, w in zip(t, [m] * k if np.ndim(m) == 0 else m)])
            assert torch.equal(got, want), (step, off, k, m)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_one_threshold_on_both_sides_of_its_lines(mkf, cuda, dtype):
    """2^20 voxels, and for FP32 fields on 16-byte boundaries 2^26: one threshold by either kernel."""
    for shape in ((64, 127, 128), (64, 129, 128), (126, 725, 728), (128, 725, 728)):
        f = make(shape, dtype, cuda)
        f = f.contiguous()
        for m in (4, 6, 1, 3, 2, 5):
            assert (mkf.field_bpfd(f, [0.25], m)[0] == plain_counts(f, 0.25, m)).all(), (shape, m)


def test_strided_fp64_on_both_sides_of_its_line(mkf, cuda):
    """6, 8 and 16 thresholds on FP64 fields with strided x, below and above 3 * 2^23 voxels."""
    import torch

    for shape in ((120, 450, 460), (130, 450, 460)):
        f = make(shape, "float64", cuda, 2)
        for k, m in ((6, 4), (8, 1), (16, 6)):
            t = np.linspace(-1.0, 1.2, k)
            got = mkf.field_bpfd(f, t, m)
            assert torch.equal(got, torch.stack([plain_counts(f, v, m) for v in t])), (shape, k)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("shape", [(90, 300, 301), (100, 300, 301)])
def test_thresholds_that_share_a_bucket(mkf, cuda, dtype, shape):
    """17 to 32 thresholds of one relation in one bucket or two of the rank table, below and above 2^23
    voxels, with elements on the thresholds and special values."""
    import torch

    f = make(shape, dtype, cuda)
    f = f.contiguous()
    for k, m in ((17, 4), (24, 6), (32, 1), (32, 3)):
        t = np.float32(300.0) + np.linspace(-1.0, 1.2, k).astype(np.float32)
        g = f + 300.0
        g.view(-1)[11::97] = float(t[k // 2])
        got = mkf.field_bpfd(g, t, m)
        for i in (0, 1, k // 2, k - 1):
            assert torch.equal(got[i], plain_counts(g, float(t[i]), m)), (k, m, i)
        assert torch.equal(got, torch.cat([mkf.field_bpfd(g, [float(v)], m) for v in t]))


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n", [14, 93, 127])
def test_batches_of_one_threshold_count(mkf, cuda, dtype, n):
    """Batches by either batched kernel (3 to 8 thresholds for every field, and with one field that differs),
    as a plan and in one shot, against the fields one at a time."""
    import torch

    fs = [make((n, n + i, n - i), dtype, cuda, 1, i) for i in range(3)]
    for k, m in ((3, 4), (5, 6), (6, 1), (8, 3)):
        for t in (np.linspace(-1.0, 1.2, k), 300.0 + 0.01 * np.arange(k)):  # (the second share a bucket)
            for ks, ms in (([t] * 3, [m] * 3), ([t, t[:1], t], [m, 2, m])):
                want = torch.cat([mkf.field_bpfd(f, v, w) for f, v, w in zip(fs, ks, ms)])
                p = mkf.BatchPlan(fs, ks, ms)
                assert torch.equal(p.launch(), want), (k, m)
                p.close()
                assert torch.equal(mkf.batch_bpfd(fs, ks, ms), want), (k, m)
