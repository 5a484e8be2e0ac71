"""Samples that only a small scale brings into the range of single precision: the
sums over a line are of in * scale."""
import numpy as np
import pytest

import crossmul as ox  # oracle/crossmul.py


@pytest.mark.gpu
@pytest.mark.parametrize("size,scale", [(3e36, 1e-34), (3e37, 1e-37)])
@pytest.mark.parametrize("looksdn", [1, 2])
@pytest.mark.parametrize("na", [20, 50, 700, 2400, 6000, 9001, 20000, 40000])
def test_large_samples_under_a_small_scale(na, looksdn, size, scale):
    import torch
    from srg_b200 import api
    rng = np.random.default_rng(na)
    # a line's sum leaves the range of 3.4e38, scale / nnn / 2 that of normal numbers
    x = [((1 + 0.3 * rng.standard_normal((4, na))) * size).astype(np.complex64) for _ in range(2)]
    scale = float(np.float32(scale))
    ig, am = api.crossmul(*[torch.from_numpy(v).cuda() for v in x], looksac=1, looksdn=looksdn, scale=scale)
    wi, wa = ox.crossmul(*x, looksac=1, looksdn=looksdn, scale=scale)
    for got, want in ((ig, wi), (am, wa)):
        got = got.cpu().numpy()
        assert np.all(np.isfinite(got.view(np.float32)))
        # the bound of the other crossmul tests
        assert np.abs(got - want).max() <= 2e-5 * np.sqrt(np.mean(np.abs(want) ** 2))
