"""4D mixed queries and steps at t next to [0, 1]: one rounding error below 0, clearly
below and clearly above.  The grid clamps the cell to its first or last time cell and
keeps the fraction (which then extrapolates), as the fp32 paths do, so the mixed kernels
that gather the 4D table are held to the mixed path's bounds: queries and predictions
within 2e-2 of the largest value of the fp32 model on the same fp16 table values,
gradients with cosine above 0.99 and within 5e-2 of the largest entry (bf16 operands
carry 8 bits of mantissa)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TIMES = [-1e-9, -0.01, 1.01]
SHAPES = [(2, 2), (4, 3)]   # features, hidden layers


def models(F, hidden):
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid4D
    from nect_b200.sampling import Geometry

    # base resolutions of 4 and 2: dense levels below the hashed ones
    enc = HashEncoderConfig(n_levels=16, n_features_per_level=F, log2_hashmap_size=13, base_resolution=4,
                            finest_resolution=160, base_resolution_t=2)
    m, ref = (HashGrid4D(enc, MLPNetConfig(n_hidden_layers=hidden), precision=p, device="cuda", seed=0)
              for p in ("mixed", "plain_fp32"))
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()
        ref.table.copy_(m.grid_table.float())
        ref.mlp.copy_(m.mlp)
    geo = Geometry(nDetector=[40, 48], dDetector=[1.5, 1.5], mode="cone", DSD=300.0, DSO=200.0, nVoxel=[32] * 3,
                   dVoxel=[1.0] * 3)
    return m, ref, geo


def off(a, b):
    return float((a - b).abs().max() / b.abs().max())


@pytest.mark.parametrize("F,hidden", SHAPES)
@pytest.mark.parametrize("t", TIMES)
def test_queries(cuda_device, F, hidden, t):
    from nect_b200.serving import query_points, reproject, slice_items, volume_items

    m, ref, geo = models(F, hidden)
    got = []
    for model in (m, ref):
        vol, sl = torch.empty(9, 16, 20, device="cuda"), torch.empty(33, 47, device="cuda")   # a stack, and not
        query_points(model, volume_items(vol, vol.shape, t))
        query_points(model, np.concatenate([slice_items(sl, sl.shape, t)]), max_blocks=7)
        got.append((vol, sl, reproject(model, geo, 0.8, t, 64), reproject(model, geo, 0.8, t, 1500)))
    for a, b in zip(*got):
        assert torch.isfinite(a).all() and off(a, b) < 2e-2, off(a, b)


@pytest.mark.parametrize("F,hidden", SHAPES)
@pytest.mark.parametrize("t", TIMES)
@pytest.mark.parametrize("staging", [False, True])
def test_steps(cuda_device, F, hidden, t, staging):
    """Without staging the backward gathers again; with it and the time slice off both halves
    and the staged scatter work on the 4D table."""
    from nect_b200 import autotune
    from nect_b200.trainer import RayBatch, Workspace, train_step

    m, ref, geo = models(F, hidden)
    P, S = geo.nDetector[0] * geo.nDetector[1], 64
    g = torch.Generator(device="cuda").manual_seed(2)
    batch = RayBatch(perm=torch.randperm(P, device="cuda", generator=g), start=0, num_rays=700, points_per_ray=S,
                     angle=0.7, max_ray_distance_per_point=geo.max_distance_traveled / S,
                     jitter=torch.rand(700, device="cuda", generator=g) - 0.5,
                     detector_offset=torch.zeros(700, 2, device="cuda"),
                     projection=torch.rand(P, device="cuda", generator=g), t=t)
    default = autotune.get_tuning()
    got = []
    try:
        autotune.set_tuning(dict(default, time_slice=0))
        for model in (m, ref):
            tg, mg = torch.zeros_like(model.table), torch.zeros_like(model.mlp)
            ws = Workspace(staging=staging)
            _, y = train_step(model, geo.get_c_geometry(), batch, geo.max_distance_traveled, tg, mg, ws, "l2")
            assert ws.error_word() == 0
            got.append((y, tg, mg))
    finally:
        autotune.set_tuning(default)
    (y, tg, mg), (yr, tgr, mgr) = got
    assert off(y, yr) < 2e-2, off(y, yr)
    for a, b in ((tg, tgr), (mg, mgr)):
        cos = float(torch.nn.functional.cosine_similarity(a.flatten().double(), b.flatten().double(), dim=0))
        assert cos > 0.99 and off(a, b) < 5e-2, (cos, off(a, b))
