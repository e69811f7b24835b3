"""The product on pairs of SMs against the product in 64 bits: edges of its tiles of 256 tokens, of its widths and of its K blocks, bands of
more than eight token tiles, several rounds of tiles, the activations of its epilogue, and the products that
`gemm_tc` gives to it by itself."""
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


FORMS = ((0, torch.float32), (1, torch.float32), (2, torch.bfloat16))           # storing, accumulating, gated


@pytest.mark.parametrize("M,N,K,there", [
    (64, 1000, 512, (0, 0, 0)), (128, 2048, 320, (0, 0, 0)), (160, 2048, 2048, (1, 1, 1)), (256, 6144, 256, (0, 0, 0)), (2048, 8192, 128, (0, 0, 1)),
    (4096, 1600, 64, (0, 0, 1)), (300, 2056, 2048, (1, 1, 1)), (2048, 2048, 6144, (1, 1, 1)), (1111, 3088, 1024, (0, 0, 0))])
def test_products_that_go_there_by_themselves(M, N, K, there):
    """Both sides of the line, and that they are on the side that is claimed here (of 148 SMs)."""
    from lia_rs_b200.kernels import ops
    _, sms = ops._device_scratch(torch.device("cuda:0"))
    for (mode, dtype), pairs in zip(FORMS, there):
        assert ops.gemm_tc_on_pairs(mode, dtype, M, N, K, sms) == bool(pairs) or sms != 148
        product(M, N, K, mode, dtype, lambda mode, a, w, out, alpha, flag: ops.gemm_tc(mode, a, w, out, alpha, flag))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K,n", [(160, 2048, 2048, None), (300, 2056, 2048, None), (257, 520, 136, 64), (600, 1000, 1000, 192), (513, 264, 72, 256)])
def test_activations(M, N, K, n, dtype):
    """The gate's ReLU, the squared ReLU and xIELU in the pair kernel's epilogue: by `gemm_tc` where it goes there by itself (n None), else in tiles of n."""
    from lia_rs_b200.kernels import ops
    _, sms = ops._device_scratch(torch.device("cuda:0"))
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(2 * N, K, device="cuda", generator=g) / K ** 0.5).to(torch.bfloat16)
    exact, constants, alpha = a.double() @ w.double().T, (0.8, 0.6), 0.5
    z = alpha * exact[:, :N]
    xielu = torch.where(z > 0, constants[0] * z * z, constants[1] * (torch.expm1(z) - z)) + 0.5 * z
    wanted = ((ops.GEMM_SWIGLU, ops.ACT_RELU, 1.0, exact[:, N:] * torch.relu(exact[:, :N])),
              (ops.GEMM_STORE, ops.ACT_RELU_SQUARED, alpha, torch.relu(z) ** 2), (ops.GEMM_STORE, ops.ACT_XIELU, alpha, xielu))
    for mode, act, scale, want in wanted:
        weights, out, flag = w if mode == ops.GEMM_SWIGLU else w[:N], torch.zeros(M, N, device="cuda", dtype=dtype), torch.zeros(1, dtype=torch.int32, device="cuda")
        if n is None:
            assert ops.gemm_tc_on_pairs(mode, dtype, M, N, K, sms)
            ops.gemm_tc(mode, a, weights, out, scale, flag, act=act, act_constants=constants)
        else:
            ops.gemm_pair(mode, a, weights, out, scale, n, flag, act=act, act_constants=constants)
        # sums of K products in 32 bits, the values of order one (off by K 2^-24), through a form whose slope is below twice the largest gate or up value; xIELU's
        # exponential by 2^-23 of itself; and half a unit of the output's type
        slope = 2.0 * max(1.0, float(exact.abs().max()))
        limit = slope * K * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20) * max(1.0, float(want.abs().max()))
        assert float((out.double() - want).abs().max()) <= limit
        assert int(flag) == 0


def test_refusals():
    from lia_rs_b200.kernels import ops
    a, w = torch.zeros(300, 64, device="cuda", dtype=torch.bfloat16), torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16)
    for n in (16, 48, 288):
        with pytest.raises(ops.KernelError):
            ops.gemm_pair(ops.GEMM_STORE, a, w, torch.zeros(300, 64, device="cuda"), 1.0, n)
    with pytest.raises(ops.KernelError):
        ops.gemm_pair(ops.GEMM_STORE, a, w, torch.zeros(300, 65, device="cuda")[:, :64], 1.0)        # rows that TMA cannot address
    for mode, act in ((ops.GEMM_ACCUM, ops.ACT_RELU_SQUARED), (ops.GEMM_SWIGLU, ops.ACT_XIELU), (ops.GEMM_STORE, ops.ACT_RELU)):
        with pytest.raises(ops.KernelError):
            ops.gemm_pair(mode, a, w, torch.zeros(300, 32 if mode == ops.GEMM_SWIGLU else 64, device="cuda"), 1.0, act=act)
    with pytest.raises(ops.KernelError):
        ops.gemm_pair(ops.GEMM_SWIGLU, a, w, torch.zeros(300, 32, device="cuda", dtype=torch.bfloat16), 1.0, 96)
