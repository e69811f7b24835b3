"""The router's product with one, two and four tokens a CTA: the same bits whatever the batch, around the lines between them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hidden,experts,extra", [(70, 3, 0), (512, 8, 1), (2048, 64, 1), (256, 128, 0)])
def test_a_batch_against_its_pieces(dtype, hidden, experts, extra):
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(hidden + experts)
    n, top = 1001, 2
    x = torch.randn(n, hidden, device="cuda", generator=g).to(dtype)
    router = torch.randn(experts + extra, hidden, device="cuda", generator=g) * hidden ** -0.5
    def route(rows):
        ids = torch.empty(len(rows), top, dtype=torch.int32, device="cuda")
        weights = torch.empty(len(rows), top, device="cuda")
        gate = torch.empty(len(rows), device="cuda") if extra else None
        ops.moe_route(rows, router, top, 1.5, ids, weights, gate)
        return [ids, weights] + ([gate] if extra else [])
    pieces = [torch.cat(parts) for parts in zip(*(route(x[at:at + 91]) for at in range(0, n, 91)))]
    for rows in (1, 148, 149, 296, 297, 299, n):
        for got, want in zip(route(x[:rows]), pieces):
            assert torch.equal(got, want[:rows]), rows
    z = x.double() @ router.double().T
    scores = z[:, :experts].softmax(dim=-1)
    assert bool((pieces[1].double() - 1.5 * scores.gather(1, pieces[0].long())).abs().max() < 1.5e-5)
