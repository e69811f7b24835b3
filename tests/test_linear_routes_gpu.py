"""Up to 256 tokens products go to the cluster kernel where it takes them, whose sums are the more exact ones; beyond, those with few output tiles and a
long K.  Both sides of the line give the product."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,cluster", [(2048, 160, 4096, True), (700, 96, 2056, True), (1000, 512, 2048, True), (1500, 512, 2048, False),
                                           (600, 256, 1024, False), (260, 1024, 4096, True), (2500, 2048, 2048, False)])
def test_few_tiles_of_a_long_k(M, N, K, cluster):
    from lia_rs_b200.kernels import ops
    from lia_rs_b200.parts import Runtime
    from lia_rs_b200.parts import linear as lin
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).to(torch.bfloat16)
    out, flag = torch.zeros(M, N, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    assert lin._few_tiles(ops.GEMM_STORE, a, w, out) == cluster
    want = a.double() @ w.double().T
    for mode, base in ((ops.GEMM_STORE, 0.0), (ops.GEMM_ACCUM, 1.0)):
        out.fill_(base)
        lin.linear(Runtime("cuda:0", torch.bfloat16), mode, a, w, out, 0.5, error_flag=flag)
        # sums of K products of order one in 32 bits
        assert float((out.double() - base - 0.5 * want).abs().max()) <= K * 2.0 ** -24 * max(1.0, float(want.abs().max())) + 2.0 ** -22
    assert int(flag) == 0


@pytest.mark.parametrize("M", [64, 128, 193, 256])
@pytest.mark.parametrize("N,K", [(1280, 1024), (520, 2048)])
def test_up_to_256_tokens_the_sums_are_the_cluster_kernels(M, N, K):
    from lia_rs_b200.kernels import ops
    from lia_rs_b200.parts import Runtime
    from lia_rs_b200.parts import linear as lin
    g = torch.Generator(device="cuda").manual_seed(M + N)
    runtime, a = Runtime("cuda:0", torch.bfloat16), torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(2 * N, K, device="cuda", generator=g) / K ** 0.5).to(torch.bfloat16)
    for mode, weights in ((ops.GEMM_STORE, w[:N]), (ops.GEMM_ACCUM, w[:N]), (ops.GEMM_SWIGLU, w)):
        out, cluster = torch.zeros(M, N, device="cuda"), torch.zeros(M, N, device="cuda")
        lin.linear(runtime, mode, a, weights, out)
        ops.gemm_cluster(mode, a, weights, cluster)
        assert torch.equal(out, cluster)
        if mode != ops.GEMM_SWIGLU:
            want = a.double() @ weights.double().T
            # an accumulator takes at most K / 8 products of the sum (four ranges and more, two accumulators each), sixteen a step, and is cut off by up to
            # 2^-23 of itself at each; the ranges' sums are then added with rounding
            assert float((out.double() - want).norm() / want.norm()) <= (K / 8 / 16 * 2.0 ** -23 + 8 * 2.0 ** -24) / 2
