"""Tiles whose pixels spread over more range bins than the staged window: the
default shape's choice by the grid's geometry, windows that widen per tile, and
the general path beyond them, against the oracle."""
import numpy as np
import pytest

import oracle as O
from helpers import phase_amp_errors
from srg_b200 import _lib, api, scene

pytestmark = pytest.mark.gpu
WIDE = [i for i in range(len(_lib.tile_configs())) if "or wide" in _lib.tile_config_name(i)]


@pytest.fixture(scope="module")
def orc():
    O.build()
    return O.Oracle()


def burst(spacing, relief, width=61, length=45, samples=2600):
    """A mini scene at the given pixel spacing (2.8 range bins per column at
    1e-4 deg), its terrain stepping by up to `relief` metres from pixel to pixel."""
    b = scene.mini_fixture(seed=41, width=width, length=length, spacing=spacing, samples=samples)
    rng = np.random.default_rng(5)
    if relief:
        b.dem = (b.dem + rng.integers(0, relief, b.dem.shape)).astype(np.int16)
    return b


def check(out, ref):
    # the split form's budget (1 mrad RMS) of the repository's other parity tests
    assert np.array_equal(out != 0, ref != 0)
    e = phase_amp_errors(out, ref)
    assert e["n"] > 100 and e["ph_rms"] < 1.0 and e["amp_rms"] < 1e-3, e


# per column 2.8, 3.6, 4.2, 5.6, 8.4, 14 and 28 bins: a 32 x 8 tile fits 128 bins up to
# about 3.4, two wide stages up to 6.8, the general path beyond; 200 m of relief
# adds about 60 bins
@pytest.mark.parametrize("relief", [0, 200])
@pytest.mark.parametrize("spacing", [1e-4, 1.3e-4, 1.5e-4, 2e-4, 3e-4, 5e-4, 1e-3])
def test_spreads(orc, spacing, relief):
    b = burst(spacing, relief)
    ref = orc.stages(b, gpu_lerp=1, gpu_scale=1, want_acc=True)["out"]
    db = api.to_device(b)
    for shear in (0, -3):
        outs = []
        for cfg in [0, -1] + WIDE:  # the wide shape is the first one's twin, to the bit
            db.out.fill_(complex(7.0, 7.0))
            api.backproject([db], tile_cfg=cfg, tile_shear=shear)
            outs.append(db.out.cpu().numpy())
            check(outs[-1], ref)
            assert np.array_equal(outs[0], outs[-1])


def test_lines_without_a_descriptor(orc):
    """Odd row strides have no TMA descriptor: the window is staged by loads."""
    import torch
    b = burst(2e-4, 200)
    ref = orc.stages(b, gpu_lerp=1, gpu_scale=1, want_acc=True)["out"]
    t = torch.zeros((b.rawdatalines, b.samples + 1), dtype=torch.complex64, device="cuda")
    t[:, :b.samples] = torch.from_numpy(b.burst).cuda()
    db = api.to_device(b, burst_tensor=t[:, :b.samples])
    outs = []
    for cfg in [0, -1]:
        api.backproject([db], tile_cfg=cfg)
        outs.append(db.out.cpu().numpy())
        check(outs[-1], ref)
    assert np.array_equal(*outs)


def test_plan_chooses_again_for_oversampled_lines(orc):
    """A plan left at the default shape takes the one for its lines: oversampled,
    a 1e-4 deg grid has 5.6 bins per column; the image is a plan's on lines
    oversampled beforehand, bit for bit."""
    import torch
    b = burst(1e-4, 0)
    db = api.to_device(b)
    plan = api.Scene([db])
    assert plan.shape() not in WIDE
    plan.set_interp(1)
    assert plan.shape() in WIDE
    s = torch.cuda.Stream()
    plan.run(stream=s.cuda_stream)
    plan.sync(stream=s.cuda_stream)
    got = db.out.cpu().numpy()
    plan.set_interp(0)
    assert plan.shape() not in WIDE
    fine = api.oversample2(db)
    api.backproject([fine], tile_shear=0)
    assert np.array_equal(got, fine.out.cpu().numpy())


@pytest.mark.parametrize("spacing,relief,samples", [(2e-4, 0, 2600), (2e-4, 200, 2601), (4e-4, 100, 2600)])
def test_dropin_on_coarse_grids(spacing, relief, samples):
    """The drop-in's kernel (lines still arriving) has the same twin: the .geo is
    the device image, to the bit."""
    import tempfile
    b = burst(spacing, relief, samples=samples)
    db = api.to_device(b)
    api.backproject([db], tile_cfg=0, tile_shear=0)
    want = db.out.cpu().numpy()
    with tempfile.TemporaryFile() as fdem, tempfile.TemporaryFile() as fout:
        fdem.write(b.dem.tobytes())
        fdem.flush()
        fout.truncate(8 * b.demwidth * b.demlength)
        api.azimuth_compress_status(b, fout.fileno(), fdem.fileno())
        got = np.memmap(fout, np.complex64, "r", shape=(b.demlength, b.demwidth))
        rows = np.array(got[db.firstline:db.firstline + db.nlines])
    merged = np.where(np.abs(want.real) > 1e-18, want, 0)
    assert np.array_equal(rows, merged)
