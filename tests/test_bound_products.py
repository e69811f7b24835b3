"""Products kept by their sizes (parts/linear.py): what is refused stays refused however often it is asked for, and what is
dropped or changes is looked up anew."""
import pytest
import torch

from lia_rs_b200.kernels import ops
from lia_rs_b200.parts import linear as module
from lia_rs_b200.parts.linear import ACCUM, STORE, linear

DTYPES = pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])


@DTYPES
def test_host_tensors_never_reach_a_kernel(dtype, monkeypatch):
    class Library:
        def __getattr__(self, name):
            raise AssertionError(f"{name} was called with host tensors")

    a, w, out = torch.zeros(40, 64, dtype=dtype), torch.zeros(24, 64, dtype=dtype), torch.zeros(40, 24)
    monkeypatch.setattr(ops, "lib", Library)
    for _ in range(3):
        with pytest.raises(ops.KernelError):
            linear(None, STORE, a, w, out)


def tensors(M, N, K, dtype, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).to(dtype)
    return a, w, torch.zeros(M, N, device="cuda")


def close(out, a, w):
    # a sum of K products: at most K roundings of a running sum no larger than a few of the results' sizes
    exact = a.double() @ w.double().T
    assert float((out.double() - exact).abs().max()) < a.shape[1] * 2.0 ** -24 * float(exact.abs().max())


@pytest.mark.gpu
@DTYPES
@pytest.mark.parametrize("M,N,K", [(40, 320, 256), (300, 24, 64)])
def test_a_kept_product_is_only_for_tensors_like_its_own(M, N, K, dtype):
    a, w, out = tensors(M, N, K, dtype)
    for _ in range(2):
        linear(None, STORE, a, w, out)
    close(out, a, w)
    crooked = torch.zeros(N, M, device="cuda").T                        # [M, N], its columns apart
    for _ in range(2):
        for args in ((a, w.cpu(), out), (a, w, out.cpu()), (a, w, crooked)):
            with pytest.raises(ops.KernelError):
                linear(None, STORE, *args)
    shifted = torch.empty(N * K + 1, device="cuda", dtype=dtype)[1:].view(N, K)      # no 16-byte loads
    shifted.copy_(w)
    for _ in range(2):
        out.zero_()
        linear(None, STORE, a, shifted, out)
        close(out, a, shifted)
    torch.cuda.synchronize()


@pytest.mark.gpu
@DTYPES
def test_dropped_products_are_looked_up_anew(dtype, monkeypatch):
    monkeypatch.setattr(module, "_MOST_BOUND", 3)
    monkeypatch.setattr(module, "_bound", {})
    for turn in range(2):
        for M in (33, 40, 50, 64, 100):
            for seed in range(2):                                       # other tensors of the same sizes
                a, w, out = tensors(M, 200, 128, dtype, seed)
                linear(None, STORE, a, w, out)
                linear(None, ACCUM, a, w, out)
                close(out / 2, a, w)
            assert len(module._bound) <= 3


@pytest.mark.gpu
def test_products_of_all_heads_are_only_for_tensors_like_their_own():
    from lia_rs_b200.parts.softmax_attention import LatentAttention
    part = LatentAttention.__new__(LatentAttention)
    B, M, N, K = 3, 40, 64, 32
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn(B, M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(B, N, K, device="cuda", generator=g).to(torch.bfloat16)
    out = torch.zeros(B, M, N, device="cuda", dtype=torch.bfloat16)
    exact = torch.einsum("bmk,bnk->bmn", a.double(), w.double())
    shifted = torch.empty(B * N * K + 1, device="cuda", dtype=torch.bfloat16)[1:].view(B, N, K)      # no 16-byte loads
    wide = torch.zeros(B, N, K + 8, device="cuda", dtype=torch.bfloat16)[:, :, :K]                   # rows that lie apart
    rounded32 = torch.zeros(B, M, N, device="cuda")
    for weight, result in ((w, out), (shifted, out), (wide, out), (w, rounded32), (w, out)):
        weight.copy_(w)
        for _ in range(2):
            result.zero_()
            part._head_products(None, a, weight, result, "k_up")
            # the result's rounding to 16 bits, and the sum's
            assert float((result.double() - exact).abs().max()) <= 2.0 ** -8 * float(exact.abs().max())
    for _ in range(2):
        for args in ((a, w.cpu(), out), (a, w.float(), out), (a, w, out[:, :-1])):
            with pytest.raises(ops.KernelError):
                part._head_products(None, *args, "k_up")
    torch.cuda.synchronize()
