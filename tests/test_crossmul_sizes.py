"""Interferogram formation at the line lengths where its transforms change: one
kernel per power of two from 64 to 8,192 points, clusters of 2, 4 and 8 CTAs for
16,384 to 65,536, cuFFT for shorter and longer lines; looks of one line down of up
to 4,096 points without scratch, everything else through the odd samples' scratch."""
import numpy as np
import pytest

import crossmul as ox  # oracle/crossmul.py

# FP32 rounding of two transforms of up to 16 levels: about 4e-7 of the line's
# RMS per sample, 5.5 sigma over 1e6 samples 2.2e-6, twice that in a product whose
# largest values are a few times its RMS.
TOL = 2e-5
WIDTHS = [1, 2, 3, 31, 32, 33, 64, 65, 127, 128, 129, 256, 257, 511, 600, 1024, 1025, 2047, 2049, 4095,
          4096, 4097, 8191, 8193, 16384, 16504, 32768, 33001, 65537]


def _images(n, nl, na, seed):
    rng = np.random.default_rng([seed, na])
    x = (rng.standard_normal((n, nl, na)) + 1j * rng.standard_normal((n, nl, na))).astype(np.complex64)
    x[:, 0, :max(1, na // 3)] = 0.0  # empty windows
    return x


def _check(got, want):
    got, want = got.cpu().numpy().astype(np.complex128), want.astype(np.complex128)
    assert got.shape == want.shape
    rms = np.sqrt(np.mean(np.abs(want) ** 2))
    assert np.abs(got - want).max() <= TOL * max(rms, 1e-30)
    assert np.array_equal(got == 0, want == 0)


@pytest.mark.gpu
@pytest.mark.parametrize("na", WIDTHS)
def test_pair_and_stack(na):
    import torch
    from srg_b200 import api
    nl = 5
    x = _images(3, nl, na, 71)
    x[2] = x[1]
    imgs = [torch.from_numpy(v).cuda() for v in x]
    imgs[2] = imgs[1]  # the same buffer twice
    for lac, ldn in [(1, 1)] + ([(3, 2), (3, 1)] if na >= 3 else []):
        want = [ox.crossmul(x[k], x[k + 1], looksac=lac, looksdn=ldn) for k in range(2)]
        ig, am = api.crossmul_stack(imgs, looksac=lac, looksdn=ldn)
        for k in range(2):
            _check(ig[k], want[k][0])
            _check(am[k], want[k][1])
        g, a = api.crossmul(imgs[0], imgs[1], looksac=lac, looksdn=ldn, scale=0.75)
        w = ox.crossmul(x[0], x[1], looksac=lac, looksdn=ldn, scale=np.float32(0.75))
        _check(g, w[0])
        _check(a, w[1])


@pytest.mark.gpu
@pytest.mark.parametrize("n,nl,na,pad", [(2, 1, 300, 3), (5, 7, 2300, 0), (66, 3, 129, 5), (4, 700, 700, 1),
                                         (9, 41, 4096, 2)])
def test_stack_runs_cut_inside_lines(n, nl, na, pad):
    """Single-look stacks whose steps are dealt in runs that start inside a
    line, with padded rows and without the mask."""
    import torch
    from srg_b200 import api
    x = _images(n, nl, na, 72)
    imgs = []
    for v in x:
        t = torch.zeros((nl, na + pad), dtype=torch.complex64, device="cuda")
        t[:, :na] = torch.from_numpy(v).cuda()
        imgs.append(t[:, :na])
    ig, am = api.crossmul_stack(imgs, looksac=1, looksdn=1, mask=False)
    for k in range(0, n - 1, max(1, n // 6)):
        w = ox.crossmul(x[k], x[k + 1], mask=False)
        _check(ig[k], w[0])
        _check(am[k], w[1])


@pytest.mark.gpu
@pytest.mark.parametrize("lac,ldn", [(2, 1), (2, 3), (4, 2), (4, 4)])
@pytest.mark.parametrize("na,pad", [(130, 0), (131, 1), (131, 0), (4600, 0), (4602, 2), (9001, 1)])
def test_looks_in_vector_loads(na, pad, lac, ldn):
    """Looks of two and four columns, with rows on 16-byte boundaries (even
    strides) and off them."""
    import torch
    from srg_b200 import api
    x = _images(2, 9, na, 73)
    imgs = []
    for v in x:
        t = torch.zeros((9, na + pad), dtype=torch.complex64, device="cuda")
        t[:, :na] = torch.from_numpy(v).cuda()
        imgs.append(t[:, :na])
    g, a = api.crossmul(*imgs, looksac=lac, looksdn=ldn)
    w = ox.crossmul(x[0], x[1], looksac=lac, looksdn=ldn)
    _check(g, w[0])
    _check(a, w[1])
