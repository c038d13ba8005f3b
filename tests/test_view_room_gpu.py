"""The column form of a view in whatever room its workspace has for sigmas: any number of
groups of 32 rays at a time gives the row form's view bit for bit, and a view that brings
its own workspace takes at most VIEW_SIGMA_BYTES for them, also where a strip of 32
detector rows has more."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def build(det, F=2):
    from nect_b200 import _lib
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid
    from nect_b200.sampling import Geometry

    geo = Geometry(nDetector=list(det), dDetector=[64.0 / det[0], 64.0 / det[1]], mode="cone", DSD=300.0, DSO=200.0,
                   nVoxel=[32] * 3, dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=16, n_features_per_level=F, log2_hashmap_size=13, base_resolution=4,
                            finest_resolution=256)
    m = HashGrid(enc, MLPNetConfig(n_hidden_layers=2), precision="mixed", device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()
    cg = geo.get_c_geometry()
    need = int(_lib.lib.nectb_train_workspace_bytes(ctypes.byref(cg.c_struct), ctypes.byref(m.grid_desc),
                                                    ctypes.byref(m.mlp_desc), det[0] * det[1]))
    return geo, m, need


@pytest.mark.parametrize("F", [2, 4])
@pytest.mark.parametrize("rays", [31, 32, 3000, 12000, 12001, 17777, 30000, 10**6])
def test_any_room_gives_the_view(cuda_device, F, rays):
    from nect_b200.serving import reproject

    geo, m, need = build((150, 200), F)
    S = 1024
    want = reproject(m, geo, 0.9, 0.0, S, workspace=torch.empty(need, dtype=torch.uint8, device="cuda"))
    room = (need + 255) // 256 * 256 + min(rays, 40000) * S * 4
    got = reproject(m, geo, 0.9, 0.0, S, workspace=torch.empty(room, dtype=torch.uint8, device="cuda"))
    assert float(want.max()) > 0.0 and torch.equal(got, want)


def test_own_workspace_is_bounded(cuda_device):
    from nect_b200.serving import VIEW_SIGMA_BYTES, reproject

    geo, m, need = build((20, 4096))
    S = 700
    assert 4 * 32 * 4096 * S > VIEW_SIGMA_BYTES
    want = reproject(m, geo, 0.9, 0.0, S, workspace=torch.empty(need, dtype=torch.uint8, device="cuda")).clone()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    got = reproject(m, geo, 0.9, 0.0, S)
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - before <= need + VIEW_SIGMA_BYTES + (2 << 20)   # and the view
    assert torch.equal(got, want)
