"""FP64 form: what a pulse that does not count holds (a stage row past a chunk's
last pulse, a position that is no number) never reaches the sum."""
import numpy as np
import pytest

import oracle as O
from helpers import rel_err
from srg_b200 import _lib, api, scene

pytestmark = pytest.mark.gpu
# the first-generation FP64 shapes: 32 x 4 takes two pulses of a pixel at a time, 32 x 8 two pixels
CFGS = [c[0] for c in _lib.tile_configs()
        if c[1] == _lib.FORM_FP64 and _lib.tile_config_name(c[0]).startswith("bp_tiles")]
# the FP64 form against the oracle: FP32 rounding of the outputs, as in the parity tests
REL = 2e-6


@pytest.fixture(scope="module")
def orc():
    O.build()
    return O.Oracle()


def burst(aperture, samples=383):
    # an odd row stride: the window is staged by bounds-checked copies
    return scene.mini_fixture(seed=51, samples=samples, aperture=aperture)


@pytest.mark.parametrize("cfg", [-1] + CFGS)
@pytest.mark.parametrize("aperture", [2, 6, 20, 25])
def test_windows_shorter_than_a_chunk(orc, aperture, cfg):
    """Tiles that span an odd number of pulses below a chunk's 32, after a launch
    that left no-number positions in every row of the stage."""
    b = burst(aperture)
    ref = orc.stages(b, gpu_lerp=1, gpu_scale=1, want_acc=True)["out"]
    db = api.to_device(b)
    before = api.to_device(burst(96))
    before.satloc.fill_(float("nan"))
    for _ in range(3):
        before.out.fill_(7.0)
        api.backproject([before], form=_lib.FORM_FP64, tile_cfg=cfg)
        api.backproject([db], form=_lib.FORM_FP64, tile_cfg=cfg)
        assert not np.any(before.out.cpu().numpy())  # no pulse in range
        out = db.out.cpu().numpy()
        assert np.array_equal(out != 0, ref != 0) and np.count_nonzero(ref) > 100
        assert rel_err(out, ref) < REL


@pytest.mark.parametrize("cfg", [-1] + CFGS)
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 1e200])
def test_positions_that_are_no_numbers(orc, bad, cfg):
    """Such a pulse is out of range for every pixel: skipped, as in the oracle."""
    b = burst(96)
    b.satloc = np.array(b.satloc, np.float64).copy()
    for k, c in [(60, 0), (61, 1), (97, 2), (130, 0), (131, 0), (132, 1), (200, 2)]:
        b.satloc[k, c] = bad
    ref = orc.stages(b, gpu_lerp=1, gpu_scale=1, want_acc=True)["out"]
    assert np.all(np.isfinite(ref.view(np.float32))) and np.count_nonzero(ref) > 100
    db = api.to_device(b)
    api.backproject([db], form=_lib.FORM_FP64, tile_cfg=cfg)
    out = db.out.cpu().numpy()
    assert np.array_equal(out != 0, ref != 0)
    assert rel_err(out, ref) < REL
