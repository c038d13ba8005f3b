"""The column form of the mixed forward (32 vertically neighbouring rays a warp)
against the row form (32 samples of one ray): the same network on the same
positions, summed in the same order, so views and predictions are equal bit for bit
and nothing has a tolerance.  Detectors whose rows do not fill a strip of 32, rays
that miss the object, sample counts that are not a multiple of a segment, one and
several strips of sigma room, a partial batch, and a batch that repeats a pixel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def build(dims, F, L=16, hidden=2, det=(150, 200), wide=1.0):
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid, HashGrid4D
    from nect_b200.sampling import Geometry

    geo = Geometry(nDetector=list(det), dDetector=[wide * 64.0 / det[0], wide * 64.0 / det[1]], mode="cone",
                   DSD=300.0, DSO=200.0, nVoxel=[32] * 3, dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=L, n_features_per_level=F, log2_hashmap_size=13, base_resolution=4,
                            finest_resolution=256, base_resolution_t=2 if dims == 4 else None)
    net = MLPNetConfig(n_hidden_layers=hidden, activation="LeakyReLU" if L == 19 else "ReLU")
    m = (HashGrid if dims == 3 else HashGrid4D)(enc, net, precision="mixed", device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()
    return geo, m


def base_workspace(geo, m):
    import ctypes

    from nect_b200 import _lib

    cg = geo.get_c_geometry()
    P = geo.nDetector[0] * geo.nDetector[1]
    return int(_lib.lib.nectb_train_workspace_bytes(ctypes.byref(cg.c_struct), ctypes.byref(m.grid_desc),
                                                    ctypes.byref(m.mlp_desc), P))


@pytest.mark.parametrize("dims,F,L,hidden,S", [(3, 2, 16, 2, 600), (4, 2, 16, 2, 601), (3, 4, 16, 3, 1024),
                                               (4, 4, 16, 2, 999), (3, 4, 19, 6, 1024)])
def test_views_are_the_same(cuda_device, dims, F, L, hidden, S):
    from nect_b200.serving import reproject

    geo, m = build(dims, F, L, hidden, wide=1.3)
    need = (base_workspace(geo, m) + 255) // 256 * 256
    strip = 4 * 32 * geo.nDetector[1] * S
    views = [reproject(m, geo, 0.9, 0.4, S, workspace=torch.empty(need + k * strip, dtype=torch.uint8, device="cuda"))
             for k in (0, 1, 2, 5)]
    views.append(reproject(m, geo, 0.9, 0.4, S))
    assert float(views[0].max()) > 0.0
    for v in views[1:]:
        assert torch.equal(v, views[0])


@pytest.mark.parametrize("F,rays,S,repeat", [(2, 30000, 333, False), (2, 20001, 512, False), (2, 30000, 333, True),
                                             (4, 30000, 512, False)])
def test_training_predictions_are_the_same(cuda_device, F, rays, S, repeat):
    """The fused step with staging (column form, encoding store) and without (row form): y_pred
    bit for bit; the staged backward reads the stored rows, so its gradients meet the
    single-pass backward's within the staged tests' 1e-5 of the largest entry."""
    from nect_b200.trainer import RayBatch, Workspace, train_step

    geo, m = build(3, F)
    P = geo.nDetector[0] * geo.nDetector[1]
    g = torch.Generator(device="cuda").manual_seed(5)
    perm = torch.randperm(P, device="cuda", generator=g)
    if repeat:
        perm[7] = perm[3]
    batch = RayBatch(perm=perm, start=0, num_rays=rays, points_per_ray=S, angle=0.3,
                     max_ray_distance_per_point=geo.max_distance_traveled / S,
                     jitter=torch.rand(rays, device="cuda", generator=g) - 0.5,
                     detector_offset=torch.zeros(rays, 2, device="cuda"),
                     projection=torch.rand(P, device="cuda", generator=g))
    got = []
    for staging in (True, False):
        tg, mg = torch.zeros_like(m.table), torch.zeros_like(m.mlp)
        loss, y = train_step(m, geo.get_c_geometry(), batch, geo.max_distance_traveled, tg, mg,
                             Workspace(staging=staging), "l2")
        got.append((y, tg, mg, float(loss)))
    assert torch.equal(got[0][0], got[1][0])
    assert abs(got[0][3] - got[1][3]) <= 1e-5 * abs(got[1][3])
    for a, b in zip(got[0][1:3], got[1][1:3]):
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())


def test_loss_of_many_rays(cuda_device):
    """The loss against float64 over the predictions.  A block adds its rays' terms once, so
    at most 4 x 148 fp32 adds meet in one number, each off by 2^-24 of it at most: a random
    walk of sqrt(592) steps of 2^-24 / 3 is 4.8e-7, and four times that is allowed."""
    from nect_b200.trainer import RayBatch, Workspace, train_step

    geo, m = build(3, 2, det=(256, 256), wide=0.5)
    P, S = 65536, 128
    g = torch.Generator(device="cuda").manual_seed(6)
    batch = RayBatch(perm=torch.randperm(P, device="cuda", generator=g), start=0, num_rays=P, points_per_ray=S,
                     angle=0.3, max_ray_distance_per_point=geo.max_distance_traveled / S,
                     jitter=torch.rand(P, device="cuda", generator=g) - 0.5,
                     detector_offset=torch.zeros(P, 2, device="cuda"),
                     projection=torch.rand(P, device="cuda", generator=g))
    tg, mg = torch.zeros_like(m.table), torch.zeros_like(m.mlp)
    loss, y = train_step(m, geo.get_c_geometry(), batch, geo.max_distance_traveled, tg, mg,
                         Workspace(staging=True), "l2")
    want = float((y.double() - batch.projection[batch.perm].double()).square().mean())
    assert abs(float(loss) - want) <= 2e-6 * want
