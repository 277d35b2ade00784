"""Measures on the device against the host's, bit for bit, for one distribution, one per CTA of the
largest grid, and more (CTAs then take several)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 22, 1184, 1185, 2500])
def test_device_measures_equal_host_for_any_count(mkf, cuda, n):
    import torch

    h = np.random.default_rng(n).integers(0, 1 << 40, size=(n, 256), dtype=np.int64)
    h[0, ::2] = 0
    got = mkf.measures_dev(torch.from_numpy(h).to(cuda)).cpu().numpy()
    assert (got == mkf.measures(h)).all()
