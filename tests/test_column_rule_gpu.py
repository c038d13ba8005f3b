"""Batches at the densities where the forward changes its form (a ray to eight pixels of a
detector of 512 rows, to four of 256, to one of fewer than 128): the predictions of the
staged step, in whichever form, are the row form's of the unstaged one bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,rays,S", [(512, 512, 32768, 192), (512, 512, 32767, 192), (256, 600, 38400, 160),
                                              (256, 600, 38399, 160), (100, 400, 40000, 160), (100, 400, 39999, 160)])
def test_predictions_do_not_depend_on_the_form(cuda_device, rows, cols, rays, S):
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid
    from nect_b200.sampling import Geometry
    from nect_b200.trainer import RayBatch, Workspace, train_step

    geo = Geometry(nDetector=[rows, cols], dDetector=[64.0 / rows, 64.0 / cols], mode="cone", DSD=300.0, DSO=200.0,
                   nVoxel=[32] * 3, dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=16, n_features_per_level=2, log2_hashmap_size=13, base_resolution=4,
                            finest_resolution=256)
    m = HashGrid(enc, MLPNetConfig(n_hidden_layers=2), precision="mixed", device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()
    P = rows * cols
    g = torch.Generator(device="cuda").manual_seed(5)
    batch = RayBatch(perm=torch.randperm(P, device="cuda", generator=g), start=0, num_rays=rays, points_per_ray=S,
                     angle=0.3, max_ray_distance_per_point=geo.max_distance_traveled / S,
                     jitter=torch.rand(rays, device="cuda", generator=g) - 0.5,
                     detector_offset=torch.zeros(rays, 2, device="cuda"),
                     projection=torch.rand(P, device="cuda", generator=g))
    got = []
    for staging in (True, False):
        tg, mg = torch.zeros_like(m.table), torch.zeros_like(m.mlp)
        got.append(train_step(m, geo.get_c_geometry(), batch, geo.max_distance_traveled, tg, mg,
                              Workspace(staging=staging), "l2")[1])
    assert float(got[0].abs().max()) > 0.0 and torch.equal(got[0], got[1])
