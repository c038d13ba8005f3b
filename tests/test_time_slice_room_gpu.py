"""Staged 4D steps in workspaces with little room beside the time slice: a batch of 2^23
sample slots or more works on the slice all the same, whose corners are half of the 4D
grid's.  Predictions are those of the recommended workspace bit for bit (the same slice);
gradients within 1e-5 of the largest entry, the bound of the staged steps against each
other (the same products, other fp32 sums)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beside_mb", [24, 96])   # of the 256 MB that a quarter of the rays stages
def test_large_batches_keep_the_time_slice(cuda_device, beside_mb):
    from nect_b200 import _lib, autotune
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid4D
    from nect_b200.sampling import Geometry
    from nect_b200.trainer import RayBatch, Workspace, train_step

    R, S, det = 32768, 256, 256
    geo = Geometry(nDetector=[det, det], dDetector=[1.0, 1.0], mode="cone", DSD=400.0, DSO=200.0, nVoxel=[64] * 3,
                   dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=16, n_features_per_level=2, log2_hashmap_size=14, base_resolution=8,
                            finest_resolution=256, base_resolution_t=2)
    m = HashGrid4D(enc, MLPNetConfig(n_hidden_layers=2), precision="mixed", device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()
    cg = geo.get_c_geometry()
    args = (ctypes.byref(cg.c_struct), ctypes.byref(m.grid_desc), ctypes.byref(m.mlp_desc), R)
    base = (int(_lib.lib.nectb_train_workspace_bytes(*args)) + 255) // 256 * 256
    default = autotune.get_tuning()

    def recommended(time_slice):
        autotune.set_tuning(dict(default, time_slice=time_slice))
        return int(_lib.lib.nectb_train_staging_bytes(*args, S))

    class Sized(Workspace):
        def get(self, *a, **k):
            self.staging = False
            super().get(*a, **k)
            if self.buf.numel() < self.size:
                self.buf = torch.empty(self.size, dtype=torch.uint8, device="cuda")
            return self.buf.data_ptr(), self.size

    g = torch.Generator(device="cuda").manual_seed(2)
    P = det * det
    batch = RayBatch(perm=torch.randperm(P, device="cuda", generator=g), start=0, num_rays=R, points_per_ray=S,
                     angle=0.7, max_ray_distance_per_point=geo.max_distance_traveled / S,
                     jitter=torch.rand(R, device="cuda", generator=g) - 0.5,
                     detector_offset=torch.zeros(R, 2, device="cuda"),
                     projection=torch.rand(P, device="cuda", generator=g), t=0.3)
    got = []
    try:
        ws = Sized()
        ws.size = base + recommended(1) - recommended(0) + (beside_mb << 20)
        for time_slice, w in ((1, ws), (1, Workspace()), (0, Workspace())):
            autotune.set_tuning(dict(default, time_slice=time_slice))
            tg, mg = torch.zeros_like(m.table), torch.zeros_like(m.mlp)
            _, y = train_step(m, cg, batch, geo.max_distance_traveled, tg, mg, w, "l2")
            assert w.error_word() == 0
            got.append((y, tg))
    finally:
        autotune.set_tuning(default)
    assert torch.equal(got[0][0], got[1][0])
    assert not torch.equal(got[0][0], got[2][0])   # the slice's fp16 rounding
    assert float((got[0][1] - got[1][1]).abs().max()) <= 1e-5 * float(got[1][1].abs().max())
