"""The composite encoder's gradient scatter for points that follow rays (each lane
walks over consecutive points) against the same points shuffled (runs merged by the
warp), and the rows written whole against one point at a time, at the edges of a
block's points.

The scatters add the same products in different orders: a table entry sums at most
n * 8 fp32 terms, whose reordering stays below 1e-5 of the largest entry (the bound
of the other reordering tests).  Rows have one order of operations: equal bit for
bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def model(F, precision):
    from nect_b200.config import HashEncoderConfig, MLPNetConfig
    from nect_b200.quadcubes import QuadCubes

    enc = HashEncoderConfig(n_levels=7, n_features_per_level=F, log2_hashmap_size=11, base_resolution=4,
                            finest_resolution=200)
    m = QuadCubes(enc, MLPNetConfig(n_hidden_layers=2, n_neurons=128, activation="LeakyReLU",
                                    output_activation="None", include_identity=True), precision=precision,
                  device="cuda", seed=3)
    with torch.no_grad():
        for k, tab in enumerate(m.tables):
            tab.normal_(0.0, 0.5, generator=torch.Generator(device="cuda").manual_seed(k))
    return m


def ray_points(n, g):
    """n consecutive samples of rays of 300 samples."""
    rays = -(-n // 300)
    a, b = (torch.rand(rays, 1, 3, device="cuda", generator=g) for _ in range(2))
    u = (torch.arange(300, device="cuda") + 0.5).view(1, -1, 1) / 300
    return (a + (b - a) * u).reshape(-1, 3)[:n].contiguous()


@pytest.mark.parametrize("F", [2, 4])
@pytest.mark.parametrize("precision", ["plain_fp32", "mixed"])
@pytest.mark.parametrize("n", [1, 17, 511, 513, 4999])
def test_walked_and_shuffled_points_agree(cuda_device, F, precision, n):
    from nect_b200.quadcubes import QuadEncode

    m = model(F, precision)
    g = torch.Generator(device="cuda").manual_seed(n)
    x = ray_points(n, g)
    t = torch.full((1,), 0.37, device="cuda")
    order = torch.randperm(n, device="cuda", generator=g)
    grads, rows = [], []
    w = torch.randn(n, m.row_width, device="cuda", generator=g)
    for pts, weight in ((x, w), (x[order].contiguous(), w[order])):
        out = QuadEncode.apply(*m.tables, m, pts, t)
        rows.append(out.detach())
        grads.append(torch.autograd.grad((out.float() * weight).sum(), list(m.tables)))
    assert torch.equal(rows[0][order], rows[1])
    one = torch.cat([QuadEncode.apply(*m.tables, m, x[i:i + 1].contiguous(), t).detach() for i in range(0, n, 97)])
    assert torch.equal(rows[0][::97], one)
    for a, b in zip(*grads):
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
