"""The word-parallel kernel at the edges of its tiles: strips of 32 (FP32) or 16 (FP64) elements and 31
row pairs, rows on and off 16-byte boundaries, one element past a strip, fields smaller than a tile,
every relation and threshold count of a pass and one more (two passes), against the oracle, exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 2), (3, 31, 17), (4, 32, 32), (3, 33, 33), (5, 63, 34), (2, 64, 65), (9, 5, 129), (70, 34, 36), (3, 40, 545)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_word_kernel_tile_edges(mkf, oracle, cuda, dtype, shape):
    import torch

    rng = np.random.default_rng(sum(shape))
    Z, Y, X = shape
    big = (rng.integers(-4, 5, size=(Z + 1, Y + 2, X + 3)) * 0.5).astype(dtype)
    big[rng.random(big.shape) < 0.02] = np.nan
    big[rng.random(big.shape) < 0.02] = np.inf
    big[rng.random(big.shape) < 0.02] = -0.0
    dev = torch.from_numpy(big).to(cuda)
    for k, rel in ((1, [4]), (2, [3, 1]), (3, [6] * 3), (4, [1, 5, 2, 4]), (5, [2, 4, 1, 6, 3]), (8, [5] * 8), (9, [4, 2] * 4 + [3])):
        t = np.sort(rng.integers(-3, 4, size=k) * 0.5)
        for off in (0, 1):
            f = np.ascontiguousarray(big[off:off + Z, off:off + Y, off:off + X])
            view = dev[off:off + Z, off:off + Y, off:off + X] if off else torch.from_numpy(f).to(cuda)
            got = mkf.field_bpfd(view, t, rel).cpu().numpy().view(np.uint64)
            want = np.stack([oracle.bpfd_field(f, (X, Y, Z), [tk], mk)[0] for tk, mk in zip(t, rel)])
            assert (got == want).all(), (k, off)
            if k <= 2:
                assert (mkf.field_bpfd_moments(view, t, rel)[0].cpu().numpy().view(np.uint64) == want).all()
            plan = mkf.BatchPlan([view, view], [t, t], [rel, rel])
            assert (plan.launch().cpu().numpy().view(np.uint64) == np.concatenate([want, want])).all()
            plan.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_one_threshold_kernels_agree(mkf, cuda, dtype):
    """The size at which one threshold moves between the two kernels (2^20 voxels, and for FP32 2^26):
    each field is counted whole and as one of two equal thresholds (always the word kernel)."""
    import torch

    for shape in ((64, 128, 127), (64, 128, 129), (127, 725, 729), (128, 725, 729)):
        f = torch.randn(shape, dtype=torch.float64, device=cuda, generator=torch.Generator(device=cuda).manual_seed(5)).to(
            torch.float32 if dtype == np.float32 else torch.float64)
        for m in (4, 6, 1, 3, 2, 5):
            one = mkf.field_bpfd(f, [0.25], m)
            two = mkf.field_bpfd(f, [0.25, 0.25], m)
            assert torch.equal(one[0], two[0]) and torch.equal(one[0], two[1])
