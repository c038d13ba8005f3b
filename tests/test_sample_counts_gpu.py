"""The windowed search for a ray's break index and the turned writes of the sampler
against the C oracle, bit for bit: sample counts around a warp, a window and its
edges, uniform and per-ray spacing, axis-aligned rays (steps of zero), large jitter
on coarse sampling, all four geometries."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N = 48
VOX = dict(sVoxel=(32.0, 32.0, 32.0), dVoxel=(1.0, 1.0, 1.0))
CYL = dict(object_radius=16.0, object_height=32.0, remove_factor_top=0.1, remove_factor_bottom=0.05)
CONE = dict(distance_source_to_origin=100.0, distance_origin_to_detector=100.0, nDetector=(N, N), dDetector=(1.5, 1.5))
PAR = dict(nDetector=(N, N), dDetector=(0.7, 0.7))


@pytest.mark.parametrize("kind,args", [("ConeGeometryVoxel", dict(CONE, **VOX)), ("ParallelGeometryVoxel", dict(PAR, **VOX)),
                                       ("ConeGeometryCylindrical", dict(CONE, **CYL)),
                                       ("ParallelGeometryCylindrical", dict(PAR, **CYL))])
@pytest.mark.parametrize("S,per_unit", [(1, 1.0), (31, 0.6), (32, 0.7), (33, 0.7), (64, 2.0), (100, 1.0), (301, 8.0),
                                        (500, 4.0)])
def test_counts_and_points_match_the_oracle(cuda_device, kind, args, S, per_unit):
    from nect_b200.sampling import ct_sampling
    from oracle import sampling as osamp

    geom = getattr(ct_sampling, kind)(**args)
    perm = torch.randperm(N * N, device=cuda_device)
    for angle, uniform in ((0.0, True), (0.7, True), (0.7, False), (1.5707964, True), (3.9, False)):
        torch.manual_seed(S)
        jitter, off = ct_sampling.draw_ray_randoms(N * N, 0.5, cuda_device)
        if angle == 0.0:
            jitter, off = torch.zeros_like(jitter), torch.zeros_like(off)
        pts, dist, counts = ct_sampling.sample_with_draws(perm, geom, angle, S, N * N, 0, 1.0 / per_unit, uniform,
                                                          jitter, off, want_counts=True)
        a = torch.tensor([angle, 0.0], dtype=torch.float32, device=cuda_device)
        c, s = torch.cos(a).cpu().numpy(), torch.sin(a).cpu().numpy()
        trig = np.array([c[0], s[0], c[1], c[1], c[1], s[1], s[1], s[1]], np.float32)
        want, wdist, wcounts = osamp.oracle_sample(osamp.to_struct(geom), perm.cpu().numpy(), 0, N * N, S, angle,
                                                   1.0 / per_unit, uniform, jitter.cpu().numpy(), off.cpu().numpy(),
                                                   trig=trig)
        np.testing.assert_array_equal(counts.cpu().numpy(), wcounts)
        np.testing.assert_array_equal(dist.cpu().numpy().view(np.uint32), wdist.view(np.uint32))
        np.testing.assert_array_equal(pts.cpu().numpy().view(np.uint32), want.view(np.uint32))
