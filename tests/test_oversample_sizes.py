"""2x oversampling of range lines at the edges of its segments: line lengths
around a segment of 1,024 samples, odd output strides (no 16-byte stores) and
the line's ends, to the bit against the taps applied one by one."""
import numpy as np
import pytest


def reference(x, h):
    """out[2k] = x[k]; out[2k+1] = sum of the 8 taps in FP32, fused as the library
    documents: h[t] (x[k-t] + x[k+1+t]) accumulated in order t = 0..3."""
    n, S = x.shape
    pad = np.zeros((n, S + 8), np.complex64)
    pad[:, 4:4 + S] = x
    out = np.zeros((n, 2 * S - 1), np.complex64)
    out[:, ::2] = x
    acc = [np.zeros((n, S - 1), np.float32) for _ in range(2)]
    for t in range(4):
        s = pad[:, 4 - t:3 - t + S] + pad[:, 5 + t:4 + t + S]
        for c, part in enumerate((s.real, s.imag)):
            # one rounding, as a fused multiply-add (exact in FP64, then rounded)
            acc[c] = (np.float64(h[t]) * part.astype(np.float64) + acc[c].astype(np.float64)).astype(np.float32)
    out[:, 1::2] = acc[0] + 1j * acc[1]
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("pad_in,pad_out", [(0, 1), (3, 0), (1, 2)])
@pytest.mark.parametrize("nsamps", [2, 3, 8, 1023, 1024, 1025, 2047, 2049, 5000])
def test_segments(nsamps, pad_in, pad_out):
    import ctypes as C
    import torch
    from srg_b200 import _lib, api
    rng = np.random.default_rng(nsamps)
    x = (rng.standard_normal((5, nsamps)) + 1j * rng.standard_normal((5, nsamps))).astype(np.complex64)
    t = torch.zeros((5, nsamps + pad_in), dtype=torch.complex64, device="cuda")
    t[:, :nsamps] = torch.from_numpy(x).cuda()
    ld = 2 * nsamps - 1 + pad_out
    out = torch.full((5, ld), 7 + 7j, dtype=torch.complex64, device="cuda")
    _lib.check(_lib.lib().srg_oversample_range_device(
        C.c_void_p(t.data_ptr()), t.stride(0), 5, nsamps, C.c_void_p(out.data_ptr()), ld, None))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    want = reference(x, api.oversample_taps())
    assert np.all(got[:, 2 * nsamps - 1:] == np.complex64(7 + 7j))
    got = got[:, :2 * nsamps - 1]
    assert np.array_equal(got[:, ::2], want[:, ::2])
    # the FP64 stand-in for the fused operation rounds twice only in a tie
    assert np.abs(got - want).max() <= 2.0 ** -22
