"""32-bit attention of few rows, a CTA a (token, query head), beside the kernel that gives each a warp (which rows of pages without 16-byte bases
go to): the same bits at the edges of its chunks of 32 and tiles of 128 keys, with a window, a list of rows and pages that are missing."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def unaligned(t):
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.reshape(-1)
    return flat[1:].view(t.shape)


@pytest.mark.parametrize("d", [16, 48, 64, 128, 144, 256])
@pytest.mark.parametrize("nq,nkv,page,window", [(4, 2, 16, None), (6, 1, 5, 100), (3, 3, 1, None)])
def test_rows_have_the_bits_of_a_warp_each(d, nq, nkv, page, window):
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(d + nq)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    positions = [0, 30, 31, 32, 127, 128, 129, 300, 511]
    blocks = 512 // page + 1
    table = torch.randperm(2 * blocks, generator=torch.Generator().manual_seed(3)).view(2, blocks).to(torch.int32).cuda()
    k, v = (torch.randn(2 * blocks, page, nkv, d, device="cuda", generator=g) for _ in range(2))
    n = len(positions)
    slots = [i % 2 for i in range(n)]
    slots[2] = -1                                                               # a row of nobody
    q = torch.randn(n, nq * d, device="cuda", generator=g)
    for rows in (None, [7, 0, -1, 8, 2]):
        results = []
        for place in (lambda t: t, unaligned):
            out = torch.full_like(q, 5.0)
            ops.attention_generic(q, place(k), place(v), ints(positions), ints(slots), table, out, nq, nkv, d, window, 0.3,
                                  rows=None if rows is None else ints(rows))
            results.append(out)
        assert torch.equal(*results)
        assert float((results[0][0] - 5.0).abs().min()) > 0 and float((results[0][2] - 5.0).abs().max()) == 0
    # keys of pages that are missing count for nothing, and the flag is up
    table[:, 40 // page] = -1
    table[:, 200 // page] = 2 * blocks
    for place in (lambda t: t, unaligned):
        flag, out = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros_like(q)
        ops.attention_generic(q, place(k), place(v), ints(positions), ints(slots), table, out, nq, nkv, d, window, 0.3, error_flag=flag)
        results.append(out)
        assert int(flag) == 2
    assert torch.equal(results[2], results[3])
