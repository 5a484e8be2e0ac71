"""The tuner's cache tells scenes apart whose default shape differs: coarse grids
and lines without a TMA descriptor, at the sizes of a fine grid on even lines."""
import pytest

from srg_b200 import _lib, api, scene

pytestmark = pytest.mark.gpu
WIDE = [i for i in range(len(_lib.tile_configs())) if "or wide" in _lib.tile_config_name(i)]


def plan(spacing, odd=False):
    import torch
    b = scene.mini_fixture(seed=61, width=61, length=45, spacing=spacing, samples=5400)
    t = None
    if odd:
        t = torch.zeros((b.rawdatalines, b.samples + 1), dtype=torch.complex64, device="cuda")
        t = t[:, :b.samples]
        t.copy_(torch.from_numpy(b.burst))
    return api.Scene([api.to_device(b, burst_tensor=t)])


def test_cache_key_sees_the_geometry():
    scenes = [dict(spacing=1e-4), dict(spacing=2e-4), dict(spacing=8e-4), dict(spacing=1e-4, odd=True)]
    wide = []
    for again in (0, 1):
        for kw in scenes:
            p = plan(**kw)
            if not again:
                wide.append(p.shape() in WIDE)
            assert p.autotune(iters=1)["from_cache"] == again, kw
            p.close()
    assert wide == [False, True, True, True]
