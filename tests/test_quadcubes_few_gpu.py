"""The composite encoder's forms for few points (blocks of eight levels, segments of four
points) against those for many, at the lines between them and at their remainders: rows
bit for bit, table gradients within 1e-5 of the largest entry (the same terms in another
order of fp32 sums, the bound of the walking tests)."""
import pytest
import torch

from test_quadcubes_walk_gpu import model, ray_points

pytestmark = pytest.mark.gpu

CHUNK = 9001   # of the form for few points


@pytest.mark.parametrize("F,precision", [(4, "mixed"), (2, "plain_fp32")])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 37632, 37633, 113152, 113153])
@pytest.mark.parametrize("loose", [False, True])
def test_few_and_many_agree(cuda_device, F, precision, n, loose):
    from nect_b200.quadcubes import QuadEncode

    m = model(F, precision)
    g = torch.Generator(device="cuda").manual_seed(n)
    x = ray_points(n, g)
    if loose:
        x = x[torch.randperm(n, device="cuda", generator=g)].contiguous()
    t = torch.full((1,), 0.37, device="cuda")
    w = torch.randn(n, m.row_width, device="cuda", generator=g)

    def run(pts, weight):
        out = QuadEncode.apply(*m.tables, m, pts, t)
        return out.detach(), torch.autograd.grad((out.float() * weight).sum(), list(m.tables))

    rows, grads = run(x, w)
    step = CHUNK if n > CHUNK else max(1, n // 3)
    parts = [run(x[i:i + step].contiguous(), w[i:i + step].contiguous()) for i in range(0, n, step)]
    assert torch.equal(rows, torch.cat([p[0] for p in parts]))
    for k, a in enumerate(grads):
        b = sum(p[1][k].double() for p in parts)
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
