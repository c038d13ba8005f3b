"""The mixed query kernel's two forms (one wide block an SM when the launch has the
GPU to itself, capped one-warpgroup blocks beside other kernels) give the same bits:
they run the same products on the same rows, so there is no tolerance.  Chunk counts
around one warpgroup, one block and one wave of a 148-SM GPU, for every model shape.
A volume (items stacked along axis 0, taken 8, 16 or 32 to a warp) gives the bits of
its slices one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,F,L,hidden", [(3, 2, 16, 2), (3, 4, 16, 3), (4, 2, 16, 2), (4, 4, 16, 3),
                                             (3, 4, 19, 6)])
@pytest.mark.parametrize("shape", [(1, 1), (1, 129), (37, 512), (333, 257)])
def test_wide_and_capped_launches_agree(cuda_device, dims, F, L, hidden, shape):
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid, HashGrid4D
    from nect_b200.serving import query_points, slice_items

    enc = HashEncoderConfig(n_levels=L, n_features_per_level=F, log2_hashmap_size=12, base_resolution=4,
                            finest_resolution=128, base_resolution_t=2 if dims == 4 else None)
    net = MLPNetConfig(n_hidden_layers=hidden, activation="LeakyReLU" if L == 19 else "ReLU")
    m = (HashGrid if dims == 3 else HashGrid4D)(enc, net, precision="mixed", device="cuda", seed=2)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(3))
        m.refresh_half()
    outs = []
    for max_blocks in (0, 3, 10_000):
        out = torch.full(shape, -1.0, device="cuda")
        query_points(m, slice_items(out, shape, 0.6, u=(0.1, 0.2, 0.9), v=(0.3, 0.8, -0.2)), max_blocks=max_blocks)
        outs.append(out)
    assert float(outs[0].min()) >= 0.0 and float(outs[0].std() if outs[0].numel() > 1 else 1.0) > 0.0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("dims,F,precision", [(3, 2, "mixed"), (4, 4, "mixed"), (3, 2, "plain_fp32"),
                                              (4, 2, "plain_fp32")])
@pytest.mark.parametrize("shape", [(7, 20, 30), (8, 3, 1), (9, 16, 16), (40, 5, 129), (65, 33, 7), (130, 11, 12)])
def test_volume_is_its_slices(cuda_device, dims, F, precision, shape):
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid, HashGrid4D
    from nect_b200.serving import query_points, volume_items

    enc = HashEncoderConfig(n_levels=16, n_features_per_level=F, log2_hashmap_size=12, base_resolution=4,
                            finest_resolution=128, base_resolution_t=2 if dims == 4 else None)
    m = (HashGrid if dims == 3 else HashGrid4D)(enc, MLPNetConfig(n_hidden_layers=2), precision=precision,
                                                device="cuda", seed=2)
    with torch.no_grad():
        m.table.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(3))
        m.refresh_half()
    whole, parts = torch.full(shape, -1.0, device="cuda"), torch.full(shape, -2.0, device="cuda")
    query_points(m, volume_items(whole, shape, 0.6, 1.5, 0.25))
    items = volume_items(parts, shape, 0.6, 1.5, 0.25)
    for i in range(shape[0]):
        query_points(m, items[i:i + 1])
    assert torch.equal(whole, parts)
    # unlike items in one call (one slice at another scale): not a stack, the same points
    mixed = torch.full(shape, -3.0, device="cuda")
    items = volume_items(mixed, shape, 0.6, 1.5, 0.25)
    items["out_scale"][-1] = 3.0
    query_points(m, items)
    assert torch.equal(whole[:-1], mixed[:-1])
