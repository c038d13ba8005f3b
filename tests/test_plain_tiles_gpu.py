"""The fp32 tile products (128 forward and 32, 64 or 128 backward samples a block)
at the edges of a tile: point counts around one tile and around a partly filled
grid, for the tilings of every model shape, against fp64 autograd on the oracle.

Forward: at most 76 + 6 * 64 fp32 products of O(1) values a point, 2^-24 each, and
the activations: 1e-5 of the largest output, the other module tests' bound.
Backward: the network without a hidden activation (with one, a pre-activation within
fp32 rounding of the kink may take either side, in any fp32 arithmetic), at most
4097 * 8 terms an entry: 1e-4 of the largest entry, the bound of the full-size smooth
step."""
import pytest
import torch

from oracle import hashgrid as ohg

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double().cpu() - b.double()).abs().max() / b.double().abs().max().clamp(min=1e-30))


SHAPES = [(3, 2, 16, 2), (4, 4, 16, 2), (3, 2, 16, 3), (4, 4, 16, 3), (3, 4, 19, 6)]


def case(dims, F, L, hidden, act, n):
    """(module, its inputs, dL/dsigma, oracle forward) of n seeded points."""
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.network import HashGrid, HashGrid4D

    enc = HashEncoderConfig(n_levels=L, n_features_per_level=F, log2_hashmap_size=10, base_resolution=4,
                            finest_resolution=64, base_resolution_t=2 if dims == 4 else None)
    m = (HashGrid if dims == 3 else HashGrid4D)(enc, MLPNetConfig(n_hidden_layers=hidden, activation=act),
                                                device="cuda", seed=4)
    g = torch.Generator().manual_seed(n)
    with torch.no_grad():
        m.table.copy_(torch.randn(m.table.shape, generator=g) * 0.5)
    x = torch.rand(n, 3, generator=g)
    dy = torch.rand(n, 1, generator=g) + 0.5
    levels, _ = ohg.layout(dims, L, 10, 4.0, float(enc.per_level_scale), 2.0 if dims == 4 else None)
    xin = x if dims == 3 else torch.cat([x, torch.full((n, 1), 0.4)], 1)
    tab = m.table.detach().cpu().double().requires_grad_()
    w = m.mlp.detach().cpu().double().requires_grad_()
    ref = ohg.mlp(ohg.encode(xin, tab, levels, 10), ohg.split_mlp_params(w, L * F, 64, hidden), act, "softplus")
    return m, (x.cuda(),) if dims == 3 else (x.cuda(), 0.4), dy, ref, tab, w


@pytest.mark.parametrize("dims,F,L,hidden", SHAPES)
@pytest.mark.parametrize("n", [1, 31, 64, 129, 4097])
def test_forward_at_tile_edges(cuda_device, dims, F, L, hidden, n):
    m, args, _, ref, _, _ = case(dims, F, L, hidden, "LeakyReLU" if L == 19 else "ReLU", n)
    assert rel(m(*args).detach(), ref.detach()) < 1e-5


@pytest.mark.parametrize("dims,F,L,hidden", SHAPES)
@pytest.mark.parametrize("n", [1, 31, 64, 129, 4097])
def test_backward_at_tile_edges(cuda_device, dims, F, L, hidden, n):
    m, args, dy, ref, tab, w = case(dims, F, L, hidden, "None", n)
    tg, mg = torch.autograd.grad(m(*args), [m.table, m.mlp], dy.cuda())
    rt, rw = torch.autograd.grad(ref, [tab, w], dy.double())
    assert rel(tg, rt) < 1e-4 and rel(mg, rw) < 1e-4
