"""The staged mixed step in workspaces below the recommended size: rounds of a quarter of
the rays beside a store of every row, of a part of them and of none, against the single
fused pass.  Predictions bit for bit (the same network on the same positions); gradients
within 1e-5 of the largest entry, the bound of the other staged-against-single-pass tests
(the same products, other fp32 sums)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_no_time_slice_without_a_round_beside_it(cuda_device):
    """A 4D step in a workspace with room for the time slice but not for a quarter of the
    rays' round beside it works on the 4D grid: the predictions of the unsliced step bit for
    bit, which the slice's fp16 rounding would change."""
    from nect_b200 import _lib, autotune
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid4D
    from nect_b200.sampling import Geometry
    from nect_b200.trainer import RayBatch, Workspace, train_step

    R, S, det = 3000, 65, (80, 96)
    geo = Geometry(nDetector=list(det), dDetector=[0.8, 0.7], mode="cone", DSD=300.0, DSO=200.0, nVoxel=[32] * 3,
                   dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=16, n_features_per_level=2, log2_hashmap_size=12, base_resolution=4,
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
    P = det[0] * det[1]
    batch = RayBatch(perm=torch.randperm(P, device="cuda", generator=g), start=0, num_rays=R, points_per_ray=S,
                     angle=0.7, max_ray_distance_per_point=geo.max_distance_traveled / S,
                     jitter=torch.rand(R, device="cuda", generator=g) - 0.5,
                     detector_offset=torch.zeros(R, 2, device="cuda"),
                     projection=torch.rand(P, device="cuda", generator=g), t=0.3)
    got = []
    try:
        ws = Sized()
        ws.size = base + recommended(1) - recommended(0) + (2 << 20)   # a quarter's round takes 6.5 MB
        for time_slice, w in ((1, ws), (0, ws), (1, Workspace())):
            autotune.set_tuning(dict(default, time_slice=time_slice))
            tg, mg = torch.zeros_like(m.table), torch.zeros_like(m.mlp)
            _, y = train_step(m, cg, batch, geo.max_distance_traveled, tg, mg, w, "l2")
            assert w.error_word() == 0
            got.append((y, tg))
    finally:
        autotune.set_tuning(default)
    assert torch.equal(got[0][0], got[1][0])
    assert not torch.equal(got[0][0], got[2][0])   # the slice, where there is room
    assert float((got[0][1] - got[1][1]).abs().max()) <= 1e-5 * float(got[1][1].abs().max())


@pytest.mark.parametrize("dims,F", [(3, 2), (3, 4), (4, 2)])
@pytest.mark.parametrize("store", [1.0, 0.4, 0.0])
def test_rows_of_small_workspaces(cuda_device, dims, F, store):
    from nect_b200 import autotune
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid, HashGrid4D
    from nect_b200.sampling import Geometry
    from nect_b200.trainer import RayBatch, Workspace, train_step

    R, S, det = 3000, 65, (80, 96)
    P, row, per_ray = det[0] * det[1], 16 * F * 2, 68 * 16 * F * 4
    geo = Geometry(nDetector=list(det), dDetector=[0.8, 0.7], mode="cone", DSD=300.0, DSO=200.0, nVoxel=[32] * 3,
                   dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=16, n_features_per_level=F, log2_hashmap_size=12, base_resolution=4,
                            finest_resolution=256, base_resolution_t=2 if dims == 4 else None)
    m = (HashGrid if dims == 3 else HashGrid4D)(enc, MLPNetConfig(n_hidden_layers=2), precision="mixed",
                                                device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()

    class Sized(Workspace):
        def get(self, model, c_geometry, num_rays, device, points_per_ray=0):
            ptr, n = super().get(model, c_geometry, num_rays, device, points_per_ray)
            less = (R - -(-R // 4)) * per_ray + (R * S - int(store * R * S)) * row   # a quarter's round, fewer rows
            return ptr, n - less - (256 if store == 0 else 0)

    g = torch.Generator(device="cuda").manual_seed(2)
    batch = RayBatch(perm=torch.randperm(P, device="cuda", generator=g), start=0, num_rays=R, points_per_ray=S,
                     angle=0.7, max_ray_distance_per_point=geo.max_distance_traveled / S,
                     jitter=torch.rand(R, device="cuda", generator=g) - 0.5,
                     detector_offset=torch.zeros(R, 2, device="cuda"),
                     projection=torch.rand(P, device="cuda", generator=g), t=0.3)
    default = autotune.get_tuning()
    got = []
    try:
        autotune.set_tuning(dict(default, time_slice=0))
        for ws in (Sized(), Workspace(staging=False)):
            tg, mg = torch.zeros_like(m.table), torch.zeros_like(m.mlp)
            _, y = train_step(m, geo.get_c_geometry(), batch, geo.max_distance_traveled, tg, mg, ws, "l2")
            assert ws.error_word() == 0
            got.append((y, tg, mg))
    finally:
        autotune.set_tuning(default)
    assert torch.equal(got[0][0], got[1][0])
    for a, b in zip(got[0][1:], got[1][1:]):
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())


@pytest.mark.parametrize("dims", [3, 4])
@pytest.mark.parametrize("shift", [8, 24])
def test_workspace_aligned_to_eight_bytes(cuda_device, dims, shift):
    """A workspace that starts on an 8-byte boundary: the same predictions bit for bit, and
    gradients within the bound above."""
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid, HashGrid4D
    from nect_b200.sampling import Geometry
    from nect_b200.trainer import RayBatch, Workspace, train_step

    class Shifted(Workspace):
        def get(self, *a, **k):
            _, n = super().get(*a, **k)
            self.whole = torch.empty(n + 64, dtype=torch.uint8, device="cuda")
            return self.whole.data_ptr() + shift, n

        def error_word(self):
            return 0   # (its address is that of the unshifted workspace)

    R, S, P = 700, 65, 40 * 48
    geo = Geometry(nDetector=[40, 48], dDetector=[1.5, 1.5], mode="cone", DSD=300.0, DSO=200.0, nVoxel=[32] * 3,
                   dVoxel=[1.0] * 3)
    enc = HashEncoderConfig(n_levels=16, n_features_per_level=2, log2_hashmap_size=12, base_resolution=4,
                            finest_resolution=256, base_resolution_t=2 if dims == 4 else None)
    m = (HashGrid if dims == 3 else HashGrid4D)(enc, MLPNetConfig(n_hidden_layers=2), precision="mixed",
                                                device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()
    g = torch.Generator(device="cuda").manual_seed(2)
    batch = RayBatch(perm=torch.randperm(P, device="cuda", generator=g), start=0, num_rays=R, points_per_ray=S,
                     angle=0.7, max_ray_distance_per_point=geo.max_distance_traveled / S,
                     jitter=torch.rand(R, device="cuda", generator=g) - 0.5,
                     detector_offset=torch.zeros(R, 2, device="cuda"),
                     projection=torch.rand(P, device="cuda", generator=g), t=0.3)
    got = []
    for ws in (Shifted(), Workspace()):
        tg, mg = torch.zeros_like(m.table), torch.zeros_like(m.mlp)
        _, y = train_step(m, geo.get_c_geometry(), batch, geo.max_distance_traveled, tg, mg, ws, "l2")
        assert ws.error_word() == 0
        got.append((y, tg, mg))
    assert torch.equal(got[0][0], got[1][0])
    for a, b in zip(got[0][1:], got[1][1:]):
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
