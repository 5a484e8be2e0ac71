"""Crossmul where the library's own transforms do not fit the device (a part of
one, say): cuFFT's take their place at every line length."""
import numpy as np
import pytest

import crossmul as ox  # oracle/crossmul.py


@pytest.fixture()
def cufft_only():
    from srg_b200 import _lib
    _lib.check(_lib.lib().srg_test_crossmul_own(0))
    yield
    _lib.check(_lib.lib().srg_test_crossmul_own(1))


@pytest.mark.gpu
@pytest.mark.parametrize("lac,ldn", [(1, 1), (2, 1), (4, 2), (3, 2)])
@pytest.mark.parametrize("na", [33, 257, 2400, 4600, 9001, 16504, 33001])
def test_stack(cufft_only, na, lac, ldn):
    import torch
    from srg_b200 import api
    rng = np.random.default_rng([na, lac])
    x = (rng.standard_normal((3, 5, na)) + 1j * rng.standard_normal((3, 5, na))).astype(np.complex64)
    x[:, 0, :na // 3] = 0.0  # empty windows
    imgs = [torch.from_numpy(v).cuda() for v in x]
    ig, am = api.crossmul_stack(imgs, looksac=lac, looksdn=ldn, scale=0.75)
    for k in range(2):
        w = ox.crossmul(x[k], x[k + 1], looksac=lac, looksdn=ldn, scale=np.float32(0.75))
        for got, want in ((ig[k], w[0]), (am[k], w[1])):
            got = got.cpu().numpy()
            rms = np.sqrt(np.mean(np.abs(want) ** 2))
            # the bound of the other crossmul tests
            assert np.abs(got.astype(np.complex128) - want).max() <= 2e-5 * rms
            assert np.array_equal(got == 0, want == 0)
