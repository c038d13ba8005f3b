"""The weight gradients of a batch that stages in three rounds (3 to 4 GiB) are no further
off than those of four rounds.  Their error is what the tensor cores' accumulators lose,
in proportion to the products between two additions to fp32 memory; three rounds add
after a quarter of the batch too, so the errors are alike up to one tile in 74 and fp32
noise: 1.15 times the four rounds' and 1e-6 of the largest entry are allowed (a third of
the batch would be 1.33 times).  The reference is the fp64 sum over sixteen parts of the
batch, each of which holds a sixteenth of the products; scaled by a power of two, a part's
gradients have the batch's bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_three_rounds_lose_no_more_than_four(cuda_device):
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid
    from nect_b200.sampling import Geometry
    from nect_b200.trainer import RayBatch, Workspace, train_step

    R, S, n, parts = 50000, 512, 256, 16
    P, per_ray = n * n, S * 32 * 4
    assert R * per_ray >> 30 == 3
    geo = Geometry(nDetector=[n, n], dDetector=[0.4, 0.4], mode="cone", DSD=300.0, DSO=200.0, nVoxel=[32] * 3,
                   dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=16, n_features_per_level=2, log2_hashmap_size=15, base_resolution=8,
                            finest_resolution=512)
    m = HashGrid(enc, MLPNetConfig(n_hidden_layers=2), precision="mixed", device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()
    g = torch.Generator(device="cuda").manual_seed(2)
    perm = torch.randperm(P, device="cuda", generator=g)
    jitter = torch.rand(R, device="cuda", generator=g) - 0.5
    projection = torch.rand(P, device="cuda", generator=g)

    class FourRounds(Workspace):
        def get(self, *a, **k):
            ptr, size = super().get(*a, **k)
            return ptr, size - (-(-R // 3) + (-R // 4)) * per_ray

    def gradient(ws, parts=1):
        tg, total = torch.zeros_like(m.table), torch.zeros_like(m.mlp, dtype=torch.float64)
        k = R // parts
        for i in range(parts):
            mg = torch.zeros_like(m.mlp)
            batch = RayBatch(perm=perm, start=i * k, num_rays=k, points_per_ray=S, angle=0.7,
                             max_ray_distance_per_point=geo.max_distance_traveled / S,
                             jitter=jitter[i * k:(i + 1) * k].contiguous(),
                             detector_offset=torch.zeros(k, 2, device="cuda"), projection=projection)
            train_step(m, geo.get_c_geometry(), batch, geo.max_distance_traveled, tg, mg, ws, "l2", 1.0 / parts)
            assert ws.error_word() == 0
            total += mg.detach().double()
        return total

    exact = gradient(Workspace(), parts)
    three, four = gradient(Workspace()), gradient(FourRounds())
    at = 0
    for size in (64 * 32, 64 * 64, 64):   # the layers
        e, top = exact[at:at + size], exact[at:at + size].abs().max()
        off3, off4 = (float((v[at:at + size] - e).abs().max() / top) for v in (three, four))
        print(f"layer at {at}: three rounds {off3:.3g}, four {off4:.3g}")
        assert off3 <= 1.15 * off4 + 1e-6, (at, off3, off4)
        at += size
