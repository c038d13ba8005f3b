"""query_points refuses graph capture (a replay would read the call's host buffer after the
allocator has given it away) and leaves stream, graph and model usable."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("given", [False, True])
def test_capture_is_refused(cuda_device, given):
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid
    from nect_b200.serving import query_points, slice_items

    enc = HashEncoderConfig(n_levels=16, n_features_per_level=2, log2_hashmap_size=13, base_resolution=4,
                            finest_resolution=160)
    m = HashGrid(enc, MLPNetConfig(n_hidden_layers=2), precision="mixed", device="cuda", seed=0)
    out, want = torch.zeros(33, 47, device="cuda"), torch.zeros(33, 47, device="cuda")
    items = slice_items(out, out.shape, 0.0)
    query_points(m, slice_items(want, want.shape, 0.0))
    torch.cuda.synchronize()
    side, graph, one = torch.cuda.Stream(), torch.cuda.CUDAGraph(), torch.zeros(1, device="cuda")
    with torch.cuda.graph(graph, stream=side):
        with pytest.raises(RuntimeError, match="captured"):
            query_points(m, items, stream=side if given else None)
        one += 1.0
    graph.replay()
    query_points(m, items)
    torch.cuda.synchronize()
    assert float(one) == 1.0 and torch.equal(out, want)
