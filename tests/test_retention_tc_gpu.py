"""Retention's portions on the tensor cores (32-bit numbers as two tf32 ones) against the recurrence in 64 bits: chunks of 128 tokens, their
blocks of 32 and what is left of them, several portions, decays from 0.3 to 1, both head sizes on either side; the error is no larger than on the 32-bit
pipes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.mark.parametrize("d,dv", [(64, 64), (128, 128), (64, 128), (128, 64)])
@pytest.mark.parametrize("lengths", [(32,), (33, 31), (65, 127, 96), (128,), (129, 40), (384, 2, 300)])
def test_portions_against_the_recurrence(d, dv, lengths):
    from lia_rs_b200.kernels import ops
    H, n, g = 40, sum(lengths), torch.Generator(device="cuda").manual_seed(d + dv + sum(lengths))
    rnd = lambda *shape: torch.randn(*shape, device="cuda", generator=g)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    decay = torch.tensor([0.3, 0.9, 1 - 2.0 ** -5, 1 - 2.0 ** -9, 1.0] * 8, device="cuda")
    rows = rnd(n, 2 * H * (d + dv) + 4)                                       # rows apart, as a padded product leaves them
    rows[:, H * d:2 * H * d] *= d ** -0.5
    slots_of, before = [2, 0, 3][:len(lengths)], rnd(4, H, d, dv)
    segments, slots, at = [], [], 0
    for slot, length in zip(slots_of, lengths):
        segments += [at, 7, length]
        slots += [slot] * length
        at += length
    chunks = ops.retention_chunks(n, len(lengths))
    results = {}
    for dtype in (torch.bfloat16, torch.float32):                              # 32-bit outputs: the 32-bit pipes
        state, out, flag = before.clone(), torch.zeros(n, H * dv, device="cuda", dtype=dtype), ints([0])
        scratch = torch.full((ops.retention_scratch_floats(chunks, H, d, dv),), float("nan"), device="cuda")
        ops.retention(rows, decay, state, ints(segments), len(lengths), chunks, ints([]), ints(slots), out, H, d, dv, 1e-5, scratch=scratch,
                      error_flag=flag)
        assert int(flag) == 0 and torch.equal(state[1], before[1])
        results[dtype] = (out.double(), state.double())
    q, k, v, gate = rows[:, :2 * H * (d + dv)].double().split([H * d, H * d, H * dv, H * dv], dim=1)
    q, k, v = q.view(n, H, d), k.view(n, H, d), v.view(n, H, dv)
    want, end = torch.empty(n, H, dv, device="cuda", dtype=F64), before.double()
    for i, slot in enumerate(slots_of):
        S = before[slot].double()
        for t in range(segments[3 * i], segments[3 * i] + lengths[i]):
            S = decay.double()[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
            want[t] = (S * q[t][:, :, None]).sum(dim=1)
        end[slot] = S
    want = (want / torch.sqrt((want * want).mean(dim=-1, keepdim=True) + 1e-5)).view(n, H * dv) * gate * torch.sigmoid(gate)
    rel = lambda a, b: float((a - b).norm() / b.norm())
    out, state = results[torch.bfloat16]
    assert float((out - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())        # rounded to bfloat16
    assert rel(out, want) <= 2.0 ** -9
    # sums of up to 384 products and their decays in 32 bits; beside the 32-bit pipes' error, which is of the same size (a fifth for the inputs' chance)
    assert rel(state, end) <= 1.2 * rel(results[torch.float32][1], end) + 2.0 ** -26 and rel(state, end) <= 4 * 2.0 ** -24
