"""The cluster product with rings of odd and even numbers of stages: widths that leave the last tile ragged, K shorter and longer than
the ring, against 64-bit; and the gated product beside two plain ones."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [17, 64, 113])
@pytest.mark.parametrize("N,K", [(6144, 2048), (6100, 512), (5630, 1032), (5640, 192), (3000, 4096)])
def test_rings_and_ragged_tiles(M, N, K):
    from lia_rs_b200.kernels import ops
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(2 * N, K, device="cuda") / math.sqrt(K)).to(torch.bfloat16)
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    gate, up = (a.double() @ part.double().T for part in (w[:N], w[N:]))
    # sums of K products of 16-bit numbers, exact in 32 bits each: K roundings of the running sum at most, in practice sqrt(K)
    most = 4 * math.sqrt(K) * 2.0 ** -24 * float(gate.abs().max())
    for part, exact in ((w[:N], gate), (w[N:], up)):
        out = torch.full((M, N), 7.0, device="cuda")
        if ops.gemm_cluster_accepts(ops.GEMM_STORE, a, part, out):
            ops.gemm_cluster(ops.GEMM_STORE, a, part, out, 1.0, flag)
            assert float((out.double() - exact).abs().max()) < most
    want = up * gate / (1 + torch.exp(-gate))
    for dtype, rounding in ((torch.float32, 2.0 ** -19), (torch.bfloat16, 2.0 ** -8)):
        out = torch.full((M, N + 4), 7.0, device="cuda", dtype=dtype)
        assert ops.gemm_cluster_accepts(ops.GEMM_SWIGLU, a, w, out[:, :N])
        ops.gemm_cluster(ops.GEMM_SWIGLU, a, w, out[:, :N], 1.0, flag)
        # (the product of two sums that are `most` off, and the result's own rounding; __expf: 2 + 1.16 |x| units in the last place)
        bound = 2 * most * (gate.abs() + up.abs() + 1) + rounding * want.abs()
        assert bool(((out[:, :N].double() - want).abs() <= bound).all())
        assert float(out[:, N:].min()) == 7.0
    torch.cuda.synchronize()
    assert flag.item() == 0
