"""The staged rank-table kernel on fields without a tensor map (rows off 16-byte boundaries, strided x):
tile edges against the oracle, and larger fields against the same data on aligned rows, exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(2, 9, 32), (3, 10, 33), (5, 17, 63), (4, 18, 95), (130, 11, 35)])
def test_ring_kernel_tile_edges(mkf, oracle, cuda, dtype, shape):
    import torch

    rng = np.random.default_rng(sum(shape))
    Z, Y, X = shape
    big = (rng.integers(-9, 10, size=(Z, Y, 2 * X + 1)) * 0.25).astype(dtype)
    for v in (np.nan, -np.nan, np.inf, -np.inf, -0.0, np.finfo(dtype).max):
        big[rng.random(big.shape) < 0.01] = v
    dev = torch.from_numpy(big).to(cuda)
    for k, m in ((5, 4), (6, 6), (8, 1), (13, 3), (16, 4)):
        t = np.linspace(-2, 2, k).round(2)
        for view, f in ((dev[:, :, 1:X + 1], big[:, :, 1:X + 1]), (dev[:, :, ::2][:, :, :X], big[:, :, ::2][:, :, :X])):
            got = mkf.field_bpfd(view, t, m).cpu().numpy().view(np.uint64)
            assert (got == oracle.bpfd_field(np.ascontiguousarray(f), (X, Y, Z), t, m)).all(), (k, m)
    assert mkf.lib().mkfKernelFaults(1) == 0


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("shape", [(200, 299, 301), (260, 361, 363)])
def test_alignment_does_not_change_counts(mkf, cuda, dtype, shape):
    import torch

    Z, Y, X = shape
    g = torch.Generator(device=cuda).manual_seed(Z)
    buf = torch.randn((Z, Y, (X + 3) // 4 * 4), dtype=torch.float64, device=cuda, generator=g).to(getattr(torch, dtype))
    aligned, tight = buf[:, :, :X], buf[:, :, :X].contiguous()
    for k in (1, 2, 3, 4, 5, 6, 12):
        for m in (4, 6):
            t = np.linspace(-1.3, 1.4, k)
            assert torch.equal(mkf.field_bpfd(aligned, t, m), mkf.field_bpfd(tight, t, m)), (k, m)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("shape", [(60, 190, 352), (130, 190, 352), (256, 512, 512)])
def test_slot_rule_sizes(mkf, cuda, dtype, shape):
    """Noise fields (cells crossing any number of the thresholds) at the sizes where a cell gets two or
    three code slots, 5 to 9 thresholds: the same counts as one threshold at a time."""
    import torch

    g = torch.Generator(device=cuda).manual_seed(shape[0])
    f = torch.randn(shape, dtype=getattr(torch, dtype), device=cuda, generator=g)
    for k, m in ((5, 4), (6, 6), (7, 1), (8, 4), (9, 3)):
        t = np.linspace(-1.1, 1.2, k)
        got = mkf.field_bpfd(f, t, m)
        assert torch.equal(got, torch.cat([mkf.field_bpfd(f, [v], m) for v in t])), (k, m)


@pytest.mark.parametrize("shape", [(128, 1023, 1023), (130, 1025, 1023)])
def test_large_fp32_fields_off_boundaries(mkf, cuda, shape):
    """Two to five thresholds of one relation below and above 2^27 voxels: the same counts as on aligned
    rows, and as one threshold at a time."""
    import torch

    Z, Y, X = shape
    g = torch.Generator(device=cuda).manual_seed(Z)
    buf = torch.randn((Z, Y, X + 1), device=cuda, generator=g)
    aligned, tight = buf[:, :, :X], buf[:, :, :X].contiguous()
    for k, m in ((1, 5), (2, 4), (3, 6), (4, 1), (5, 3), (5, 4)):
        t = np.linspace(-1.3, 1.4, k)
        got = mkf.field_bpfd(tight, t, m)
        assert torch.equal(got, mkf.field_bpfd(aligned, t, m)), (k, m)
        assert torch.equal(got, torch.cat([mkf.field_bpfd(tight, [v], m) for v in t])), (k, m)
