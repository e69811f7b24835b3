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
    pairs, (tile_rows, pad) = ids.numel(), ops.moe_pair_tile_rows(128 * experts, experts)
    assert (tile_rows, pad) == (256, 32)
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


@pytest.mark.parametrize("n", [16, 64, 256, 257])
def test_a_shared_experts_sums_are_those_of_its_products_alone(n):
    """Up to 256 tokens the cluster kernel's (or the few-token kernel's), more exact than a pair's one accumulator; beyond, one accumulator either way."""
    from lia_rs_b200.cache import CacheManager
    from lia_rs_b200.engine import StepEntry, StepRuntime
    from lia_rs_b200.kernels import ops
    from lia_rs_b200.parts import FEED_FORWARDS, Runtime, linear as lin
    g = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *shape: (torch.randn(*shape, device="cuda", generator=g) * shape[-1] ** -0.5).to(torch.bfloat16)
    h, ff, ffs, experts = 1024, 64, 2048, 4
    tensors = {"L.router": rnd(experts, h), "L.shared.gate": rnd(ffs, h), "L.shared.up": rnd(ffs, h), "L.shared.down": rnd(h, ffs)}
    for e in range(experts):                                                 # the routed experts add nothing
        tensors.update({f"L.e{e}.gate": rnd(ff, h), f"L.e{e}.up": rnd(ff, h), f"L.e{e}.down": torch.zeros(h, ff, device="cuda", dtype=torch.bfloat16)})
    runtime = Runtime("cuda:0", torch.bfloat16)
    part = FEED_FORWARDS["expert_mixture"](dict(hidden=h, experts=experts, top=2, intermediate=ff, shared={"intermediate": ffs}, shared_gated=False),
                                           tensors, "L.", runtime)
    cache = CacheManager({}, {}, 32, 16, 1, 512, torch.bfloat16, "cuda:0")
    steps, slot = StepRuntime(cache, 1000, 512, "cuda:0"), cache.admit()
    assert cache.ensure(slot, 0, n)
    x = (rnd(n, h).float() * h ** 0.5).to(torch.bfloat16)
    out, act, want = torch.zeros(n, h, device="cuda"), torch.empty(n, ffs, device="cuda", dtype=torch.bfloat16), torch.zeros(n, h, device="cuda")
    part.forward(steps.begin([StepEntry(slot, [1] * n, 0, [])]), x, out, 1.0, store=True)
    steps.finish()
    alone = (lambda *product: lin.linear(runtime, *product)) if n <= 256 else ops.gemm_pair
    alone(lin.SWIGLU, x, part.w_shared_gate_up, act)
    alone(lin.STORE, act, part.w_shared_down, want)
    assert torch.equal(out, want)
