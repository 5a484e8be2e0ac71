"""Range compression over the pulse lengths where its path changes: segments of
8,192 samples with few or many valid ones, and cuFFT's padded rows beyond them."""
import numpy as np
import pytest

import rangecomp as orc  # oracle/rangecomp.py

FS = 64.345


@pytest.mark.gpu
@pytest.mark.parametrize("npts,nsamps", [(1, 40), (2, 8192), (643, 8193), (3371, 3372), (4096, 24000), (4097, 24001),
                                         (5147, 29001), (6434, 9000), (6860, 32768), (6900, 32768),
                                         (8192, 8200), (8193, 9000), (20000, 32768)])
def test_matches_oracle(npts, nsamps):
    import torch
    from srg_b200 import api
    pulse = dict(samplefreq=FS, startfreq=-20.2, ramprate=40.8 * FS / npts,
                 pulselength=float(np.float32((npts + 0.5) / FS)))
    assert orc.replica(**pulse)[1] == npts
    rng = np.random.default_rng([npts, nsamps])
    x = (rng.standard_normal((5, nsamps)) + 1j * rng.standard_normal((5, nsamps))).astype(np.complex64)
    want = orc.range_compress(x, **pulse)
    got = api.range_compress(torch.from_numpy(x).cuda(), **pulse).cpu().numpy()
    assert got.shape == want.shape == (5, nsamps - npts)
    # FP32 rounding of two 13-level transforms (about 4e-7 RMS, 6 sigma), as the
    # bound of the other range-compression tests
    rms = np.sqrt(np.mean(np.abs(want) ** 2))
    assert np.abs(got.astype(np.complex128) - want).max() / rms < 2e-5
