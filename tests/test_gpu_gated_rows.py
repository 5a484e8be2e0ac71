"""A burst whose lines are still arriving: no row is read before it is announced,
also where a chunk goes through two wide stages, which read a row more."""
import ctypes as C

import numpy as np
import pytest

from srg_b200 import _lib, api, scene

pytestmark = pytest.mark.gpu
BASE = 64


def gated(db, word, cfg):
    import torch
    o = _lib.default_options(_lib.FORM_SPLIT)
    o.tile_cfg, o.tile_shear, o.spin_limit = cfg, 0, 4096
    d = db.desc()
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = _lib.lib().srg_bp_burst_device_gated(C.byref(d), C.c_void_p(word.data_ptr()), BASE, 1,
                                              C.byref(o), st)
    assert rc == _lib.SRG_OK, _lib.last_error()
    rc = _lib.lib().srg_sync_check(st)
    assert rc in (_lib.SRG_OK, _lib.SRG_E_TIMEOUT), _lib.last_error()
    return rc == _lib.SRG_OK


def rows_awaited(db, cfg):
    """The fewest announced rows with which the call completes."""
    import torch
    word = torch.empty((1,), dtype=torch.int32, device="cuda")
    lo, hi = 0, db.b.rawdatalines  # waits run out with lo, not with hi
    while hi - lo > 1:
        mid = (lo + hi) // 2
        word.fill_(BASE + mid)
        lo, hi = (lo, mid) if gated(db, word, cfg) else (mid, hi)
    return hi


@pytest.mark.parametrize("samples", [2600, 2601])  # with and without a TMA descriptor
@pytest.mark.parametrize("spacing,more", [(1e-4, 0), (2e-4, 1)])
def test_rows_awaited(samples, spacing, more):
    """One tile column, whose chunks fit the first shape's window (31 pulses, 31 rows)
    or take two stages of 16 rows each."""
    b = scene.mini_fixture(seed=71, width=32, length=16, spacing=spacing, samples=samples, aperture=60,
                           dem_kind="flat")
    db = api.to_device(b)
    narrow, wide = rows_awaited(db, 0), rows_awaited(db, -1)
    assert 60 < narrow < b.rawdatalines - 1
    assert wide == narrow + more
    # and with those rows the image is the ungated one
    import torch
    word = torch.full((1,), BASE + wide, dtype=torch.int32, device="cuda")
    db.out.fill_(complex(7.0, 7.0))
    assert gated(db, word, -1)
    got = db.out.cpu().numpy()
    api.backproject([db], tile_shear=0)
    assert np.array_equal(got, db.out.cpu().numpy()) and np.count_nonzero(got) > 100
