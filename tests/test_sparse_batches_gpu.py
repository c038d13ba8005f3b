"""Batches of few rays on a detector of many pixels: the scheduler skips the empty pixels
between them and finds every ray.  A ray's prediction does not depend on the batch, so it
equals the one of a batch of all pixels bit for bit (fp32 path, and the mixed path without
staging), and each ray adds its share of the gradient: the gradients of a batch and of
its rays one by one agree within 1e-5 of the largest entry (fp32 sums in another order)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DET = (131, 127)
P = DET[0] * DET[1]
PICKS = {"first": [0], "last": [P - 1], "ends": [P - 1, 0], "neighbours": [700, 701, 702, 733, 734],
         "a strip apart": list(range(5, P, 32)), "31 and 33 apart": [64, 95, 128, 5000, 5031, 5064, P - 32, P - 1],
         "many": list(range(0, P, 7))}


@pytest.mark.parametrize("precision", ["plain_fp32", "mixed"])
@pytest.mark.parametrize("pick", PICKS)
def test_every_ray_is_found(cuda_device, precision, pick):
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid
    from nect_b200.sampling import Geometry
    from nect_b200.trainer import RayBatch, Workspace, train_step

    geo = Geometry(nDetector=list(DET), dDetector=[0.5, 0.5], mode="cone", DSD=300.0, DSO=200.0, nVoxel=[32] * 3,
                   dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=16, n_features_per_level=2, log2_hashmap_size=12, base_resolution=4,
                            finest_resolution=256)
    m = HashGrid(enc, MLPNetConfig(n_hidden_layers=2), precision=precision, device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        if precision == "mixed":
            m.refresh_half()
    projection = torch.rand(P, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    S = 48

    def step(pixels, tg, mg, scale=1.0):
        perm = torch.tensor(pixels, dtype=torch.int64, device="cuda")
        n = perm.numel()
        batch = RayBatch(perm=perm, start=0, num_rays=n, points_per_ray=S, angle=0.7,
                         max_ray_distance_per_point=geo.max_distance_traveled / S,
                         jitter=torch.zeros(n, device="cuda"), detector_offset=torch.zeros(n, 2, device="cuda"),
                         projection=projection)
        ws = Workspace(staging=False)
        _, y = train_step(m, geo.get_c_geometry(), batch, geo.max_distance_traveled, tg, mg, ws, "l2", scale)
        assert ws.error_word() == 0
        return y

    pixels = PICKS[pick]
    all_y = step(list(range(P)), torch.zeros_like(m.table), torch.zeros_like(m.mlp))
    tg, mg = torch.zeros_like(m.table), torch.zeros_like(m.mlp)
    y = step(pixels, tg, mg)
    assert torch.equal(y, all_y[torch.tensor(pixels, device="cuda")])
    if len(pixels) <= 8:
        t1, m1 = torch.zeros_like(m.table), torch.zeros_like(m.mlp)
        for p in pixels:
            step([p], t1, m1, 1.0 / len(pixels))
        for a, b in ((tg, t1), (mg, m1)):
            assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
