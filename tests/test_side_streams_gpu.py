"""Views and time slices on a stream of the caller's: their buffers belong to that stream,
so allocations and writes on the current stream right after the call (while the call has
not begun) do not reach them.  Bit for bit the view of the current stream."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def build():
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid4D
    from nect_b200.sampling import Geometry

    enc = HashEncoderConfig(n_levels=16, n_features_per_level=2, log2_hashmap_size=13, base_resolution=4,
                            finest_resolution=160, base_resolution_t=2)
    m = HashGrid4D(enc, MLPNetConfig(n_hidden_layers=2), precision="mixed", device="cuda", seed=0)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(1))
        m.refresh_half()
    geo = Geometry(nDetector=[128, 130], dDetector=[0.5, 0.5], mode="cone", DSD=250.0, DSO=160.0, nVoxel=[32] * 3,
                   dVoxel=[1.0] * 3)
    return m, geo


@pytest.mark.parametrize("kwargs", [{}, {"pixels": (11, 9001)}, {"warpgroups": 3}])
@pytest.mark.parametrize("S", [64, 640])   # rows, and the column form with its sigma room
def test_views_on_a_side_stream(cuda_device, kwargs, S):
    from nect_b200.serving import reproject

    m, geo = build()
    want = torch.zeros(128 * 130, device="cuda")
    reproject(m, geo, 0.8, 0.6, S, out=want, **kwargs)
    begin, count = kwargs.get("pixels", (0, want.numel()))
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)   # the view starts some 10 ms after the writes below
    view = reproject(m, geo, 0.8, 0.6, S, stream=side, **kwargs)
    junk = []
    for mib in (1, 2, 4, 8, 16, 64, 256, 300) * 2:
        junk.append(torch.full((mib << 18,), float("nan"), device="cuda"))
    torch.cuda.synchronize()
    assert torch.equal(view.flatten()[begin:begin + count], want[begin:begin + count])


def test_time_slice_on_a_side_stream(cuda_device):
    from nect_b200.serving import time_slice

    m, _ = build()
    want = time_slice(m, 0.3)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
    got = time_slice(m, 0.3, stream=side)
    junk = [torch.full((1 << k,), 7, dtype=torch.uint8, device="cuda") for k in range(16, 26)]
    torch.cuda.synchronize()
    assert torch.equal(got, want) and len(junk) == 10
