"""The staged gradient scatter (a lane marching over a ray's samples) against the
single-pass backward's per-sample scatter, where segments, rows of four samples
and detector strips have remainders: S not a multiple of 4 or of a segment, a
detector whose rows do not fill a strip, a repeated pixel (batch order), 2 and 4
features, 3D, the 4D time slice and the 16-corner 4D scatter.

Both scatter the same dL/d(encoding) (the same bf16 network on the same rows), so
the table gradients differ by the order of fp32 sums: a largest entry of at most
N = 2^17 terms each off by 2^-24 of it at most, in practice sqrt(N) 2^-24 = 2.2e-5
of the absolute sum; 1e-5 of the largest entry is the bound the other
staged-against-single-pass tests use."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def grads(m, geo, S, rays, staging, repeat, seed=2):
    from nect_b200.trainer import RayBatch, Workspace, train_step

    P = geo.nDetector[0] * geo.nDetector[1]
    g = torch.Generator(device="cuda").manual_seed(seed)
    perm = torch.randperm(P, device="cuda", generator=g)
    if repeat:
        perm[1] = perm[0]
    batch = RayBatch(perm=perm, start=0, num_rays=rays, points_per_ray=S, angle=0.7,
                     max_ray_distance_per_point=geo.max_distance_traveled / S,
                     jitter=torch.rand(rays, device="cuda", generator=g) - 0.5,
                     detector_offset=torch.zeros(rays, 2, device="cuda"),
                     projection=torch.rand(P, device="cuda", generator=g), t=0.3)
    tg, mg = torch.zeros_like(m.table), torch.zeros_like(m.mlp)
    train_step(m, geo.get_c_geometry(), batch, geo.max_distance_traveled, tg, mg, Workspace(staging=staging), "l2")
    return tg


@pytest.mark.parametrize("dims,F,S,det,rays,repeat,time_slice", [
    (3, 2, 1, (33, 5), 165, False, 1),
    (3, 2, 31, (40, 7), 280, False, 1),
    (3, 2, 33, (31, 9), 100, True, 1),
    (3, 4, 66, (65, 4), 260, False, 1),
    (4, 2, 130, (33, 6), 33, False, 1),
    (4, 2, 37, (33, 6), 198, False, 0),
    (4, 4, 95, (32, 8), 250, False, 0),
])
def test_march_matches_per_sample_scatter(cuda_device, dims, F, S, det, rays, repeat, time_slice):
    from nect_b200 import autotune
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid, HashGrid4D
    from nect_b200.sampling import Geometry

    geo = Geometry(nDetector=list(det), dDetector=[50.0 / det[0], 50.0 / det[1]], mode="cone", DSD=300.0, DSO=200.0,
                   nVoxel=[32] * 3, dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=16, n_features_per_level=F, log2_hashmap_size=12, base_resolution=4,
                            finest_resolution=256, base_resolution_t=2 if dims == 4 else None)
    m = (HashGrid if dims == 3 else HashGrid4D)(enc, MLPNetConfig(n_hidden_layers=2), precision="mixed",
                                                device="cuda", seed=0)
    with torch.no_grad():
        g = torch.Generator(device="cuda").manual_seed(1)
        m.table.copy_(torch.randn(m.table.shape, device="cuda", generator=g) * 0.3)
        m.refresh_half()
    default = autotune.get_tuning()
    try:
        # the time slice rounds the blended table to fp16: compare like with like
        autotune.set_tuning(dict(default, time_slice=time_slice))
        staged = grads(m, geo, S, rays, True, repeat)
        if time_slice and dims == 4:
            autotune.set_tuning(dict(default, time_slice=0))
            single = grads(m, geo, S, rays, True, repeat)
            bound = 2e-2   # fp16 slice rounding (the time-slice tests' bound)
        else:
            single = grads(m, geo, S, rays, False, repeat)
            bound = 1e-5
    finally:
        autotune.set_tuning(default)
    assert float((staged - single).abs().max()) <= bound * float(single.abs().max())
