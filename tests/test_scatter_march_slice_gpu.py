"""The staged march of a 4D batch against the single-pass backward's per-sample scatter:
on the 4D grid at an inner t, and on the time slice at t = 0 and t = 1, where the blend is
one of its two time vertices and the fp16 slice holds the table's own values, so nothing
is rounded again.  Both scatter the same dL/d(encoding) (the same bf16 network on the same
rows): table gradients within 1e-5 of the largest entry, the bound of the other
staged-against-single-pass tests, and predictions bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F,S,det,rays", [(2, 130, (33, 6), 33), (2, 37, (33, 6), 198), (4, 95, (32, 8), 250)])
@pytest.mark.parametrize("t,time_slice", [(0.3, 0), (0.0, 1), (1.0, 1)])
def test_march_matches_per_sample_scatter(cuda_device, F, S, det, rays, t, time_slice):
    from nect_b200 import autotune
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid4D
    from nect_b200.sampling import Geometry
    from nect_b200.trainer import RayBatch, Workspace, train_step

    geo = Geometry(nDetector=list(det), dDetector=[50.0 / det[0], 50.0 / det[1]], mode="cone", DSD=300.0, DSO=200.0,
                   nVoxel=[32] * 3, dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=16, n_features_per_level=F, log2_hashmap_size=12, base_resolution=4,
                            finest_resolution=256, base_resolution_t=2)
    m = HashGrid4D(enc, MLPNetConfig(n_hidden_layers=2), precision="mixed", device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()
    P = det[0] * det[1]
    g = torch.Generator(device="cuda").manual_seed(2)
    batch = RayBatch(perm=torch.randperm(P, device="cuda", generator=g), start=0, num_rays=rays, points_per_ray=S,
                     angle=0.7, max_ray_distance_per_point=geo.max_distance_traveled / S,
                     jitter=torch.rand(rays, device="cuda", generator=g) - 0.5,
                     detector_offset=torch.zeros(rays, 2, device="cuda"),
                     projection=torch.rand(P, device="cuda", generator=g), t=t)
    default = autotune.get_tuning()
    got = []
    try:
        autotune.set_tuning(dict(default, time_slice=time_slice))
        for staging in (True, False):   # the unstaged step has no slice
            tg, mg = torch.zeros_like(m.table), torch.zeros_like(m.mlp)
            _, y = train_step(m, geo.get_c_geometry(), batch, geo.max_distance_traveled, tg, mg,
                              Workspace(staging=staging), "l2")
            got.append((y, tg))
    finally:
        autotune.set_tuning(default)
    assert float(got[1][1].abs().max()) > 0.0 and torch.equal(got[0][0], got[1][0])
    assert float((got[0][1] - got[1][1]).abs().max()) <= 1e-5 * float(got[1][1].abs().max())
