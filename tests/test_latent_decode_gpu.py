"""The tensor-core kernel for attention in a latent's space and the putting together of up to 64 ranges of which some see no key,
against 64-bit."""
import pytest
import torch

import plain_vatunex as pv
from test_vatunex_parts_gpu import Pages, dev, ints

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.mark.parametrize("heads,rank,dr,window", [(1, 64, 16, None), (17, 192, 48, 70), (2, 448, 128, 129), (16, 512, 64, None), (5, 480, 64, 33)])
def test_ranges_put_together(heads, rank, dr, window):
    from lia_rs_b200.kernels import ops
    g = torch.Generator().manual_seed(rank + dr)
    dtype, T = torch.bfloat16, 300
    cache = Pages(2, T, 16, seed=7)
    q = (torch.randn(T, heads, rank + dr, generator=g, dtype=F64) * 2).to(dtype)
    k = torch.randn(T, 1, rank + dr, generator=g, dtype=F64).to(dtype)
    latent_pages, part_pages = cache.empty(1, rank, dtype), cache.empty(1, dr, dtype)
    cache.fill(latent_pages, 1, k[:, :, :rank])
    cache.fill(part_pages, 1, k[:, :, rank:])
    where = [0, 1, 31, 32, 33, 63, 64, 127, 200, 256, 299, 5]
    slots = [1] * (len(where) - 1) + [-1]                                  # the last row belongs to nobody
    n, scale = len(where), (rank + dr) ** -0.5
    q_here = q[where]
    q1 = dev(q_here[:, :, :rank].transpose(0, 1).contiguous(), dtype)
    q2 = dev(q_here[:, :, rank:].reshape(n, heads * dr).contiguous(), dtype)
    want = pv.softmax_attention(q.to(F64), k.to(F64), k.to(F64)[:, :, :rank], scale, window=window)[where][:-1]
    for splits in (1, 2, 5, 33, 64):
        out = torch.zeros(heads, n, rank, dtype=dtype, device="cuda")
        words = splits * heads * n * (rank + 2)
        # (scratch that begins 8 bytes past a 16-byte boundary, and holds what a range without keys must not pass on)
        partial = torch.full((words + 2,), float("nan"), device="cuda")[2:] if splits > 1 else None
        ops.latent_attention(q1, q2, latent_pages, part_pages, ints(where), ints(slots), cache.table, out, heads, window, scale,
                             splits=splits, partial=partial)
        got = out.float().cpu().to(F64).transpose(0, 1)
        assert float(got[-1].abs().max()) == 0.0
        # the probabilities and the result are rounded to bfloat16 (eight bits: each by at most 2^-8 of itself), and what the
        # probabilities lose stands against a sum that may cancel: |sum dp v| <= 2^-8 sum p |v|
        bound = 2.0 ** -8 * (want.abs() + pv.softmax_attention(q.to(F64), k.to(F64), k.to(F64)[:, :, :rank].abs(), scale, window=window)[where][:-1])
        assert bool(((got[:-1] - want).abs() <= 1.02 * bound + 1e-6).all()), splits
