"""Products of many tokens with few output tiles and a long K go to the cluster kernel; both sides of the line give the product."""
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
