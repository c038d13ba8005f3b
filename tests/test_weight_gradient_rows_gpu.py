"""The staged backward adds its weight gradients four values at a time where the caller's
buffer is 16-byte aligned, one by one elsewhere: both give the same gradients (the same
sums in another order of fp32 additions: 1e-5 of the largest entry, the bound of the
staged-against-single-pass tests), next to untouched neighbours."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F,L,hidden", [(2, 16, 2), (4, 16, 2), (2, 16, 3), (4, 19, 6)])
def test_unaligned_weight_gradients(cuda_device, F, L, hidden):
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid
    from nect_b200.sampling import Geometry
    from nect_b200.trainer import RayBatch, Workspace, train_step

    geo = Geometry(nDetector=[40, 48], dDetector=[1.5, 1.5], mode="cone", DSD=300.0, DSO=200.0, nVoxel=[32] * 3,
                   dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=L, n_features_per_level=F, log2_hashmap_size=12, base_resolution=4,
                            finest_resolution=256)
    m = HashGrid(enc, MLPNetConfig(n_hidden_layers=hidden, activation="LeakyReLU" if L == 19 else "ReLU"),
                 precision="mixed", device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()
    P, R, S = 40 * 48, 700, 64
    g = torch.Generator(device="cuda").manual_seed(2)
    batch = RayBatch(perm=torch.randperm(P, device="cuda", generator=g), start=0, num_rays=R, points_per_ray=S,
                     angle=0.7, max_ray_distance_per_point=geo.max_distance_traveled / S,
                     jitter=torch.rand(R, device="cuda", generator=g) - 0.5,
                     detector_offset=torch.zeros(R, 2, device="cuda"),
                     projection=torch.rand(P, device="cuda", generator=g))
    got = []
    for shift in (0, 1, 2, 3):
        buf = torch.zeros(m.mlp.numel() + 8, device="cuda")
        tg, mg = torch.zeros_like(m.table), buf[shift:shift + m.mlp.numel()]
        ws = Workspace()
        train_step(m, geo.get_c_geometry(), batch, geo.max_distance_traveled, tg, mg, ws, "l2")
        assert ws.error_word() == 0
        assert not buf[:shift].any() and not buf[shift + m.mlp.numel():].any()
        got.append(mg.clone())
    assert float(got[0].abs().max()) > 0.0
    for v in got[1:]:
        assert float((v - got[0]).abs().max()) <= 1e-5 * float(got[0].abs().max())
