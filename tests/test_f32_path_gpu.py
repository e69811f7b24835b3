"""The 32-bit path's tiled kernels against the kernels for every size: the same chains of additions, so the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def unaligned(t):
    """The same numbers where no 16-byte load can read them: the kernel for every size serves such operands."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.reshape(-1)
    return flat[1:].view(t.shape)


@pytest.mark.parametrize("M,N,K", [(1, 4, 4), (8, 96, 20), (16, 33, 16), (33, 31, 68), (47, 130, 100), (64, 64, 48), (129, 257, 36),
                                   (600, 1024, 64), (700, 1290, 132), (1300, 2050, 32), (2500, 515, 16)])
def test_tiled_product_has_the_bits_of_the_kernel_for_every_size(M, N, K):
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, w = torch.randn(M, K, device="cuda", generator=g), torch.randn(2 * N, K, device="cuda", generator=g)
    before = torch.randn(M, N, device="cuda", generator=g)
    for mode, weights, act in [(ops.GEMM_STORE, w[:N], 0), (ops.GEMM_ACCUM, w[:N], 0), (ops.GEMM_SWIGLU, w, 0),
                               (ops.GEMM_SWIGLU, w, ops.ACT_RELU)]:
        got, want = before.clone(), before.clone()
        ops.gemm_simt(mode, a, weights, got, 0.75, act=act)
        ops.gemm_simt(mode, unaligned(a), unaligned(weights), want, 0.75, act=act)
        assert torch.equal(got, want), (mode, act)


def test_tiled_batched_product_with_strides():
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(37, 5, 24, device="cuda", generator=g).transpose(0, 1)           # [5, 37, 24], a head's rows apart
    w = torch.randn(5, 50, 24, device="cuda", generator=g)
    got, want = (torch.zeros(37, 5, 50, device="cuda").transpose(0, 1) for _ in range(2))
    ops.gemm_simt_batched(ops.GEMM_STORE, a, w, got)
    ops.gemm_simt_batched(ops.GEMM_STORE, a, unaligned(w), want)
    assert torch.equal(got, want)


@pytest.mark.parametrize("d", [32, 64, 96, 128])
@pytest.mark.parametrize("nq,nkv,page", [(2, 2, 16), (8, 1, 5), (16, 2, 16), (6, 2, 1), (64, 1, 7)])
def test_prompt_attention_has_the_bits_of_the_kernel_for_every_size(d, nq, nkv, page):
    """Portions of 2 tokens to several tiles, from position 0 and late, on three requests; later positions of the pages hold
    what no token may see (infinities and NaN among it)."""
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(d + nq)
    portions = [(0, 0, 2), (1, 31, 33), (2, 5, 140), (0, 300, 65)]              # slot, first position, tokens
    slots_n, longest = 4, 400
    blocks = (longest + page - 1) // page
    order = torch.randperm(slots_n * blocks, generator=torch.Generator().manual_seed(1))
    table = order.view(slots_n, blocks).to(torch.int32).cuda()
    k_pages, v_pages = (torch.randn(slots_n * blocks, page, nkv, d, device="cuda", generator=g) for _ in range(2))
    for run in portions:
        slot, start, count = run
        for cut in (portions[:1], portions[1:2], portions[2:3], portions[3:], portions[1:]):
            if run not in cut:
                continue
            positions = [p for s, first, n in cut for p in range(first, first + n)]
            slot_ids = [s for s, first, n in cut for _ in range(n)]
            segments, at = [], 0
            for s, first, n in cut:
                segments += [at, first, n]
                at += n
            ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
            q = torch.randn(at, nq * d, device="cuda", generator=g)
            v_here = v_pages.clone()
            for s, first, n in cut:                                             # behind the portion's end
                end = first + n
                v_here[int(table[s, end // page]), end % page, :, ::2] = float("nan")
                v_here[int(table[s, end // page]), end % page, :, 1::2] = float("inf")
            got, want = (torch.zeros(at, nq * d, device="cuda") for _ in range(2))
            per_tile = ops.attention_prefill_f32_tokens_per_tile(nq // nkv, d)
            tiles = sum((n + per_tile - 1) // per_tile for _, _, n in cut)
            ops.attention_prefill_f32(q, k_pages, v_here, ints(segments), len(cut), tiles, ints(slot_ids), table, got, nq, nkv, d, 0.3)
            ops.attention_generic(q, k_pages, v_here, ints(positions), ints(slot_ids), table, want, nq, nkv, d, None, 0.3)
            assert torch.equal(got, want), (run, float((got - want).abs().max()))


def test_a_missing_page_is_flagged_and_reads_nothing():
    from lia_rs_b200.kernels import ops
    q = torch.randn(8, 64, device="cuda")
    pages = torch.randn(4, 4, 1, 64, device="cuda")
    table = torch.tensor([[2, -1, 9]], dtype=torch.int32, device="cuda")
    flag, out = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(8, 64, device="cuda")
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    ops.attention_prefill_f32(q, pages, pages, ints([0, 0, 8]), 1, 1, ints([0] * 8), table, out, 1, 1, 64, 1.0, error_flag=flag)
    assert int(flag) == 2
    # token t attends over keys 0 .. min(t, 3) of page 2 alone: sums of 64 products and of four, their exponentials' scores off by as much
    k = pages[2, :, 0].double()
    for t in range(8):
        seen = k[:min(t, 3) + 1]
        want = torch.softmax(seen @ q[t].double(), dim=0) @ seen
        assert float((out[t].double() - want).abs().max()) < 64 * 2.0 ** -23 * float((k.abs() @ q[t].double().abs()).max())


def test_operands_without_16_byte_bases_go_to_the_kernel_for_every_size():
    from types import SimpleNamespace
    from lia_rs_b200.parts.paged_attention import PagedAttention
    g = torch.Generator(device="cuda").manual_seed(5)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    nq, nkv, d, n = 4, 2, 32, 70
    pages = torch.randn(2, 30, 5, nkv, d, device="cuda", generator=g)
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    segments = [(0, 0, n - 1, 0), (1, 20, 1, n - 1)]
    ctx = SimpleNamespace(n_tokens=n, n_prefill_segments=1, segments=segments, prefill_segments=ints([0, 0, n - 1]), error_flag=flag,
                          slots=ints([0] * (n - 1) + [1]), positions=ints(list(range(n - 1)) + [20]), decode_rows=ints([n - 1]))
    table = torch.arange(30, dtype=torch.int32, device="cuda").view(2, 15)
    attention = PagedAttention(torch.float32, nq, nkv, d, None, 0.3)
    q = torch.randn(n, nq * d, device="cuda", generator=g)
    want = torch.zeros_like(q)
    aligned_kv = SimpleNamespace(k_pages=pages[0], v_pages=pages[1], block_table=table)
    attention.forward(ctx, q, aligned_kv, want)
    for shifted in ("q", "k", "v", "out"):
        place = lambda name, t: unaligned(t) if name == shifted else t
        kv = SimpleNamespace(k_pages=place("k", pages[0]), v_pages=place("v", pages[1]), block_table=table)
        out = place("out", torch.zeros_like(q))
        attention.forward(ctx, place("q", q), kv, out)
        assert torch.equal(out, want), shifted
    assert int(flag) == 0
