"""Few long rays are sampled in parts by several warps: positions, distances and counts of
five rays alone equal those of the same rays in a batch that fills the GPU, bit for bit,
for every geometry and sample counts around the parts' edges."""
import pytest
import torch

pytestmark = pytest.mark.gpu

VOX = dict(nVoxel=[64] * 3, dVoxel=[1.0] * 3)
GEOMETRIES = {
    "cone": dict(mode="cone", DSD=300.0, DSO=200.0, **VOX),
    "parallel": dict(mode="parallel", **VOX),
    "cylinder": dict(mode="cone", DSD=300.0, DSO=200.0, reconstruction_mode="cylindrical", **VOX),
}


@pytest.mark.parametrize("kind", GEOMETRIES)
@pytest.mark.parametrize("S", [64, 65, 511, 1023, 1024, 1025, 4096, 4099])
def test_parts_equal_whole_rays(cuda_device, kind, S):
    from nect_b200.sampling import Geometry, ct_sampling

    geo = Geometry(nDetector=[60, 50], dDetector=[1.3, 1.4], **GEOMETRIES[kind])
    R, few = 1400, 5
    g = torch.Generator(device="cuda").manual_seed(3)
    perm = torch.randperm(3000, device="cuda", generator=g)
    jitter = torch.rand(R, device="cuda", generator=g) - 0.5
    offset = torch.rand(R, 2, device="cuda", generator=g) - 0.5

    def sample(n):
        return ct_sampling.sample_with_draws(perm, geo.get_c_geometry(), 0.7, S, n, 0, geo.max_distance_traveled / S,
                                             True, jitter[:n].contiguous(), offset[:n].contiguous())

    many, alone = sample(R), sample(few)
    assert len(many) == len(alone) >= 2
    for a, b in zip(alone, many):
        assert torch.equal(a, b[:few])
    assert bool((alone[0] != 0).any())
