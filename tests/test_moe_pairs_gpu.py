"""The experts' products on pairs of SMs, the shared expert's in the same launch, against 64 bits: experts without rows, with one, with rows
around the 32 that a warp stores and the 256 of a tile; widths that are no multiples of the tiles'."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,shared", [((1, 0, 3), 0), ((31, 32, 33, 0), 5), ((255, 256, 257), 300), ((0, 700), 64), ((2,) * 40, 0)])
@pytest.mark.parametrize("N,K,N2,K2", [(40, 72, 200, 136), (256, 64, 96, 200)])
def test_grouped_and_plain_product_in_one_launch(rows, shared, N, K, N2, K2):
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(sum(rows) + N)
    rnd = lambda *shape: torch.randn(*shape, device="cuda", generator=g)
    experts = len(rows)
    ids = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(rows)])
    ids = ids[torch.randperm(len(ids), generator=torch.Generator().manual_seed(1))].cuda()
    pairs, (tile_rows, pad) = ids.numel(), ops.moe_pair_tile_rows(12 * experts, experts)
    assert (tile_rows, pad) == (256, 32) and ops.moe_pair_tile_rows(4 * experts - 1, experts) == (0, 0)
    ints = lambda n: torch.full((n,), -7, dtype=torch.int32, device="cuda")
    max_tiles, cap = ops.moe_max_tiles(pairs, experts, tile_rows), ops.moe_padded_rows(pairs, experts, pad)
    offsets, order, inverse, tiles, n_tiles = ints(experts + 1), ints(cap), ints(pairs), ints(3 * max_tiles), ints(1)
    ops.moe_plan(ids, experts, offsets, order, inverse, tiles, n_tiles, tile_rows, pad=pad)
    x = rnd(pairs, K).to(torch.bfloat16)
    sorted_x = torch.empty(cap, K, device="cuda", dtype=torch.bfloat16)
    ops.moe_gather(x, order, 1, sorted_x)
    x2 = rnd(shared, K2).to(torch.bfloat16)
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    for mode, act, dtype in ((ops.GEMM_SWIGLU, 0, torch.bfloat16), (ops.GEMM_STORE, 0, torch.float32), (ops.GEMM_STORE, ops.ACT_RELU_SQUARED, torch.bfloat16)):
        double = 2 if mode == ops.GEMM_SWIGLU else 1
        w = (rnd(experts, double * N, K) / K ** 0.5).to(torch.bfloat16)
        w2 = (rnd(double * N2, K2) / K2 ** 0.5).to(torch.bfloat16)
        out, out2 = torch.zeros(cap, N, device="cuda", dtype=dtype), torch.zeros(shared, N2, device="cuda", dtype=dtype)
        ops.gemm_pair_grouped(mode, sorted_x, w, out, tiles, n_tiles, max_tiles, pairs, (x2, w2, out2) if shared else None, error_flag=flag, act=act)

        def form(z, width):
            if mode == ops.GEMM_SWIGLU:
                return z[:, width:] * z[:, :width] * torch.sigmoid(z[:, :width])
            return torch.relu(z) ** 2 if act else z
        # sums of K products in 32 bits, the values of order one (their squares' size for the squared form), rounded to the output's type
        want = torch.cat([form(x[p:p + 1].double() @ w[int(e)].double().T, N) for p, e in enumerate(ids.tolist())])
        limit = lambda v: (2 * 200 * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0)) * max(1.0, float(v.abs().max()))
        assert float((out[inverse.long()].double() - want).abs().max()) <= limit(want)
        if shared:
            want = form(x2.double() @ w2.double().T, N2)
            assert float((out2.double() - want).abs().max()) <= limit(want)
    assert int(flag) == 0
