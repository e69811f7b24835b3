"""The experts' rows put together four elements a thread, beside the kernel that takes any width and alignment: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", [4, 132, 1024, 2052])
@pytest.mark.parametrize("top", [1, 2, 5, 8])
@pytest.mark.parametrize("own", [None, torch.float32, torch.bfloat16])
def test_fours_against_single_elements(hidden, top, own):
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(hidden + top)
    n, rows = 37, 64
    y = torch.randn(rows * hidden + 1, device="cuda", generator=g)
    inverse = torch.randint(0, rows, (n, top), device="cuda", generator=g, dtype=torch.int32)
    inverse[::3, 0] = -1                                                  # identity outputs, or nothing without `x`
    weights = torch.rand(n, top, device="cuda", generator=g)
    shared, gate = torch.randn(n, hidden, device="cuda", generator=g), torch.rand(n, device="cuda", generator=g)
    x = None if own is None else torch.randn(n, hidden + 6, device="cuda", generator=g).to(own)[:, 3:3 + hidden].contiguous()
    before = torch.randn(n, hidden, device="cuda", generator=g)
    for store in (True, False):
        for shared_y, shared_gate in [(None, None), (shared, None), (shared, gate)]:
            results = []
            for shift in (0, 1):                                          # rows of `y` that 16-byte loads can read, and that they can't
                flat = torch.zeros_like(y)
                part = flat[shift:shift + rows * hidden].view(rows, hidden)
                part.copy_(y[:rows * hidden].view(rows, hidden))
                residual = before.clone()
                ops.moe_combine(residual, part, inverse.view(-1), weights, shared_y, shared_gate, top, 0.75, store, x=x)
                results.append(residual)
            assert torch.equal(*results)
            # and the sum itself, in 64-bit: every choice, the shared rows and what was there are one rounding each
            chosen = y[:rows * hidden].view(rows, hidden).double()[inverse.clamp(min=0).long()]
            mine = torch.zeros(n, hidden, device="cuda", dtype=torch.float64) if x is None else x.double()
            chosen = torch.where((inverse >= 0)[:, :, None], chosen, mine[:, None, :]) * weights.double()[:, :, None]
            terms = [chosen]
            if shared_y is not None:
                terms.append((shared.double() * (gate.double()[:, None] if shared_gate is not None else 1.0))[:, None, :])
            terms = torch.cat(terms, dim=1) * 0.75
            want = terms.sum(dim=1) + (0.0 if store else before.double())
            size = terms.abs().sum(dim=1) + (0.0 if store else before.double().abs())
            assert bool(((results[0].double() - want).abs() <= (top + 3) * 2.0 ** -24 * size + 1e-30).all())
