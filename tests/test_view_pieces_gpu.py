"""Pieces of a view at the default warpgroups: any range of pixels (fewer than a row, a
part of a row at the end, one pixel, the whole view) in the default workspace and in one
with room to spare gives the whole view's pixels bit for bit (the same network on the
same positions, so nothing has a tolerance; with the time slice off, which a larger
workspace of a 4D model would otherwise take)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

COLS = 40


@pytest.mark.parametrize("dims,F", [(3, 2), (4, 2), (3, 4)])
@pytest.mark.parametrize("extra", [0, 1 << 20, 64 << 20])
@pytest.mark.parametrize("piece", [1, 17, COLS, 500, 48 * COLS])
def test_pieces_are_the_view(cuda_device, dims, F, extra, piece):
    from nect_b200 import autotune
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid, HashGrid4D
    from nect_b200.sampling import Geometry
    from nect_b200.serving import reproject, reproject_workspace_bytes

    enc = HashEncoderConfig(n_levels=16, n_features_per_level=F, log2_hashmap_size=13, base_resolution=4,
                            finest_resolution=160, base_resolution_t=2 if dims == 4 else None)
    m = (HashGrid if dims == 3 else HashGrid4D)(enc, MLPNetConfig(n_hidden_layers=2), precision="mixed",
                                                device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()
    geo = Geometry(nDetector=[48, COLS], dDetector=[1.2, 1.2], mode="cone", DSD=250.0, DSO=160.0, nVoxel=[32] * 3,
                   dVoxel=[1.0] * 3)
    P, S = 48 * COLS, 64
    default = autotune.get_tuning()
    try:
        autotune.set_tuning(dict(default, time_slice=0))
        whole = reproject(m, geo, 0.8, 0.6, S).flatten()
        out = torch.full((P,), float("nan"), device="cuda")
        # not a multiple of the row, so that pieces start inside one; the first 20 pieces of the smallest
        for begin in range(0, min(P, 20 * piece), piece):
            count = min(piece, P - begin)
            ws = torch.empty(reproject_workspace_bytes(m, geo, count) + extra, dtype=torch.uint8, device="cuda")
            reproject(m, geo, 0.8, 0.6, S, out=out, workspace=ws, pixels=(begin, count))
    finally:
        autotune.set_tuning(default)
    n = min(P, 20 * piece)
    assert float(whole.max()) > 0.0
    assert torch.equal(out[:n], whole[:n]) and torch.isnan(out[n:]).all()
