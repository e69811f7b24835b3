"""The product on pairs of SMs against the product in 64 bits: edges of its tiles of 256 tokens, of its widths and of its K blocks, bands of
more than eight token tiles, several rounds of tiles, and the products that `gemm_tc` gives to it by itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def product(M, N, K, mode, dtype, launch, pad=0):
    """`launch(mode, a, w, out, alpha, flag)` against 64 bits; rows of `out` lie `pad` elements apart, which stay as they are."""
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K + mode)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(2 * N if mode == ops.GEMM_SWIGLU else N, K, device="cuda", generator=g) / K ** 0.5).to(torch.bfloat16)
    wide = torch.randn(M, N + pad, device="cuda", generator=g).to(dtype)
    before, flag = wide.clone(), torch.zeros(1, dtype=torch.int32, device="cuda")
    launch(mode, a, w, wide[:, :N], 0.5, flag)
    exact = a.double() @ w.double().T
    if mode == ops.GEMM_SWIGLU:
        want = exact[:, N:] * exact[:, :N] * torch.sigmoid(exact[:, :N])
    else:
        want = 0.5 * exact + (before[:, :N].double() if mode == ops.GEMM_ACCUM else 0)
    # sums of K products in 32 bits, the values of order one: below K 2^-24 of their size, and half a unit of the output's type
    limit = (K * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20)) * max(1.0, float(want.abs().max()))
    assert float((wide[:, :N].double() - want).abs().max()) <= limit
    assert int(flag) == 0 and (pad == 0 or torch.equal(wide[:, N:], before[:, N:]))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (128, 32, 64), (129, 264, 72), (256, 256, 512), (257, 520, 136), (600, 1000, 1000), (2300, 40, 64),
                                   (2560, 2080, 192)])
def test_tiles_of_every_width(M, N, K, dtype):
    from lia_rs_b200.kernels import ops
    for mode in (ops.GEMM_STORE, ops.GEMM_SWIGLU) + ((ops.GEMM_ACCUM,) if dtype == torch.float32 else ()):
        for n in range(64, 257, 64) if mode == ops.GEMM_SWIGLU else range(32, 257, 32):
            product(M, N, K, mode, dtype, lambda mode, a, w, out, alpha, flag: ops.gemm_pair(mode, a, w, out, alpha, n, flag), pad=8)


@pytest.mark.parametrize("M,N,K", [(64, 1000, 512), (128, 2048, 320), (160, 2048, 2048), (256, 6144, 256), (2048, 8192, 128), (4096, 1600, 64)])
def test_products_that_go_there_by_themselves(M, N, K):
    from lia_rs_b200.kernels import ops
    for mode, dtype in ((ops.GEMM_STORE, torch.float32), (ops.GEMM_ACCUM, torch.float32), (ops.GEMM_SWIGLU, torch.bfloat16)):
        product(M, N, K, mode, dtype, lambda mode, a, w, out, alpha, flag: ops.gemm_tc(mode, a, w, out, alpha, flag))


def test_refusals():
    from lia_rs_b200.kernels import ops
    a, w = torch.zeros(300, 64, device="cuda", dtype=torch.bfloat16), torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16)
    for n in (16, 48, 288):
        with pytest.raises(ops.KernelError):
            ops.gemm_pair(ops.GEMM_STORE, a, w, torch.zeros(300, 64, device="cuda"), 1.0, n)
    with pytest.raises(ops.KernelError):
        ops.gemm_pair(ops.GEMM_STORE, a, w, torch.zeros(300, 65, device="cuda")[:, :64], 1.0)        # rows that TMA cannot address
    with pytest.raises(ops.KernelError):
        ops.gemm_pair(ops.GEMM_SWIGLU, a, w, torch.zeros(300, 32, device="cuda", dtype=torch.bfloat16), 1.0, 96)
