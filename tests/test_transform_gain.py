"""The transforms' constants are rounded to one side; what that takes from every
result is put back: crossmul's and range compression's mean gain and error against
64 bits."""
import numpy as np
import pytest

import crossmul as OX
import rangecomp as ORC
from srg_b200 import api

pytestmark = pytest.mark.gpu


def gain(got, want):
    got, want = np.asarray(got, np.complex128).ravel(), want.ravel()
    return abs(np.sum((got - want) * want.conj()) / np.sum(np.abs(want) ** 2))


def rel(got, want):
    return np.linalg.norm(np.asarray(got, np.complex128) - want) / np.linalg.norm(want)


def images(rows, na, seed):
    """Two images that share most of their signal, without unformed samples."""
    rng = np.random.default_rng(seed)
    z = rng.standard_normal((3, rows, na, 2)).astype(np.float32).view(np.complex64)[..., 0]
    return z[0] + np.float32(0.5) * z[1], z[0] + np.float32(0.5) * z[2]


# Uncorrected, the odd samples are short by 0.75e-7, 0.9e-7, 1.0e-7, 1.3e-7 at 1,024,
# 2,048, 4,096 and 8,192 points and a product of both images by twice that on its odd
# half: the products' gain is off by as much.  The correction's step is 1.2e-7, so
# half of it may remain.
@pytest.mark.parametrize("looksdn", [1, 2])
@pytest.mark.parametrize("na", [900, 1700, 2400, 4000, 6000, 9001, 20000, 40000])
def test_crossmul_gain(na, looksdn):
    import torch
    a, b = images(24, na, na)
    ig, am = api.crossmul(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), looksac=1,
                          looksdn=looksdn)
    wi, wa = OX.crossmul(a, b, 1, looksdn, dtype=np.complex128)
    assert gain(ig.cpu().numpy(), wi) < 6e-8
    assert gain(am.cpu().numpy(), wa) < 6e-8


def test_crossmul_error_of_single_looks():
    """Lines of 2,049-4,096 samples: no further from 64 bits than self-sorting
    transforms with a factor per bin, whose error was 1.40e-7."""
    import torch
    a, b = images(64, 2400, 7)
    ig, am = api.crossmul(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), looksac=1, looksdn=1)
    wi, wa = OX.crossmul(a, b, 1, 1, dtype=np.complex128)
    assert rel(ig.cpu().numpy(), wi) < 1.40e-7
    assert rel(am.cpu().numpy(), wa) < 1.40e-7


@pytest.mark.parametrize("pulse_us", [20.0, 52.4, 80.0])
def test_range_compression_gain_and_error(pulse_us):
    """Uncorrected the fused filter's results are short by 1.0e-7 (the tables' part
    of the gain, a few 1e-8 to either side, stays); self-sorting transforms erred
    by 2.01e-7 on pulses of 3,371 samples."""
    import torch
    args = (64.345, -20.2, 40.8 / pulse_us, pulse_us)
    x = images(12, 24000, int(pulse_us))[0]
    got = api.range_compress(torch.from_numpy(x).cuda(), *args)
    rep, npts = ORC.replica(*args)
    X = np.fft.fft(x.astype(np.complex128), n=ORC.RANFFT, axis=1)
    want = np.fft.ifft(X * np.fft.fft(rep.astype(np.complex128)).conj(), axis=1) * ORC.RANFFT
    got, want = got.cpu().numpy()[:, :24000 - npts], want[:, :24000 - npts]
    assert gain(got, want) < 4e-8
    assert rel(got, want) < 2.01e-7
