"""Pairs with more lines than the chip holds at once: every CTA, and every cluster of
the longer lines, takes several lines in turn, from both images, the last turn
not for all of them."""
import numpy as np
import pytest

import crossmul as ox  # oracle/crossmul.py


@pytest.mark.gpu
@pytest.mark.parametrize("na,nl,lac,ldn", [
    (50, 12001, 1, 2), (200, 6003, 2, 2), (700, 1601, 1, 2), (3000, 701, 2, 2),  # several lines of a CTA, or one
    (4600, 701, 1, 2), (8000, 601, 1, 1),                                        # 8,192 points
    (9001, 331, 1, 1), (16384, 331, 2, 1), (16504, 203, 1, 1), (32001, 203, 4, 2),  # clusters of 2 and 4
    (33001, 101, 1, 1), (60000, 151, 1, 1)])                                        # of 8
def test_lines_taken_in_turn(na, nl, lac, ldn):
    import torch
    from srg_b200 import api
    rng = np.random.default_rng([na, nl])
    imgs = []
    for _ in range(2):
        t = torch.from_numpy(rng.standard_normal((nl, na, 2), dtype=np.float32)).cuda()
        imgs.append(torch.view_as_complex(t))
    ig, am = api.crossmul(*imgs, looksac=lac, looksdn=ldn)
    again = api.crossmul(*imgs, looksac=lac, looksdn=ldn)
    assert torch.equal(torch.view_as_real(ig), torch.view_as_real(again[0]))
    assert torch.equal(torch.view_as_real(am), torch.view_as_real(again[1]))
    # every line in 64 bits on the device
    nnn, nout, ncol = ox.fft_length(na), nl // ldn, na // lac
    for r in range(0, nout, 32):
        rows = slice(r * ldn, min(r + 32, nout) * ldn)
        up = []
        for x in imgs:
            X = torch.fft.fft(x[rows].to(torch.complex128), n=nnn, dim=1)
            U = torch.zeros((X.shape[0], 2 * nnn), dtype=torch.complex128, device="cuda")
            U[:, :nnn // 2] = X[:, :nnn // 2]
            U[:, 2 * nnn - nnn // 2:] = X[:, nnn // 2:]
            up.append(torch.fft.ifft(U, dim=1)[:, :2 * na])

        def looks(v):
            v = v.reshape(-1, ldn, na, 2).sum(3).sum(1)[:, :ncol * lac]
            return v.reshape(-1, ncol, lac).sum(2)

        g = looks(up[0] * up[1].conj())
        a = torch.complex(looks(up[0].abs() ** 2).sqrt(), looks(up[1].abs() ** 2).sqrt())
        for got, want in ((ig[r:r + 32], g), (am[r:r + 32], a)):
            rms = want.abs().square().mean().sqrt()
            # the bound of the other crossmul tests
            assert (got - want).abs().max() <= 2e-5 * rms, (r, na)
    # and the oracle on the first and last rows
    for r in (0, nout - 1):
        x = [v[r * ldn:(r + 1) * ldn].cpu().numpy() for v in imgs]
        wi, wa = ox.crossmul(*x, looksac=lac, looksdn=ldn)
        for got, want in ((ig[r], wi), (am[r], wa)):
            rms = np.sqrt(np.mean(np.abs(want) ** 2))
            assert np.abs(got.cpu().numpy() - want).max() <= 2e-5 * rms
