"""The decays' product with a thread a channel and eight tokens beside the kernel for every rank and alignment: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,H,d,dv,rank", [(1, 2, 8, 4, 8), (9, 3, 30, 20, 16), (64, 16, 16, 32, 24), (1030, 5, 64, 32, 16), (17, 1, 300, 16, 40)])
def test_encode_rows_has_the_bits_of_the_kernel_for_every_rank(n, H, d, dv, rank, dtype):
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(n + d)
    rows = torch.randn(n, 2 * H * (d + dv) + rank + 3, device="cuda", generator=g)
    flat = (torch.randn(H * d * rank + 1, device="cuda", generator=g) * 0.3).to(dtype)
    bias = torch.randn(H * d, device="cuda", generator=g)
    slots = torch.arange(n, dtype=torch.int32, device="cuda") % 3 - 1            # every third row is nobody's
    results = []
    for crooked in (False, True):
        w = flat[1:].view(H * d, rank) if crooked else flat[1:].clone().view(H * d, rank)
        mine, log_decay = rows.clone(), torch.full((n, H * d), 7.0, device="cuda")
        ops.gla_encode(mine, w, bias, log_decay, slots, H, d, dv, 0.4, 16.0)
        results.append((mine, log_decay))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    nobody = slots < 0
    assert torch.equal(results[0][0][nobody], rows[nobody]) and float((results[0][1][nobody] - 7.0).abs().max()) == 0
