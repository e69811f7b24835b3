"""What retention's prompt portions (heads of 64 or 128 elements) keep at every size: bfloat16 outputs are the 32-bit outputs rounded, a portion's bits
do not depend on the other portions of its step, and a value that is not finite stays out of the tokens ahead of it (those that its warp's sixteen
tokens do not hold)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
H = 24


def step(rows, lengths, d, dv, before, dtype):
    from lia_rs_b200.kernels import ops
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    segments, slots, at = [], [], 0
    for slot, length in enumerate(lengths):
        segments += [at, 7, length]
        slots += [slot] * length
        at += length
    chunks = ops.retention_chunks(at, len(lengths))
    scratch = torch.empty(ops.retention_scratch_floats(chunks, H, d, dv), device="cuda")
    decay = torch.tensor([0.4, 0.97, 1 - 2.0 ** -9, 1.0] * (H // 4), device="cuda")
    state, out = before.clone(), torch.zeros(at, H * dv, device="cuda", dtype=dtype)
    ops.retention(rows, decay, state, ints(segments), len(lengths), chunks, ints([]), ints(slots), out, H, d, dv, 1e-5, scratch=scratch)
    return out, state


def inputs(n, d, dv, portions):
    g = torch.Generator(device="cuda").manual_seed(n + d + dv)
    rows = torch.randn(n, 2 * H * (d + dv), device="cuda", generator=g)
    rows[:, H * d:2 * H * d] *= d ** -0.5
    return rows, torch.randn(portions, H, d, dv, device="cuda", generator=g)


@pytest.mark.parametrize("d,dv", [(64, 64), (128, 128), (64, 128), (128, 64)])
@pytest.mark.parametrize("lengths", [(2,), (64,), (129, 200), (300, 2, 65)])
def test_outputs_of_either_type_and_portions_alone_have_the_same_bits(d, dv, lengths):
    rows, before = inputs(sum(lengths), d, dv, len(lengths))
    out, state = step(rows, lengths, d, dv, before, torch.float32)
    rounded, again = step(rows, lengths, d, dv, before, torch.bfloat16)
    assert torch.equal(rounded, out.to(torch.bfloat16)) and torch.equal(again, state)
    at = 0
    for i, length in enumerate(lengths):
        for dtype, whole in ((torch.float32, out), (torch.bfloat16, rounded)):
            alone, end = step(rows[at:at + length], (length,), d, dv, before[i:i + 1], dtype)
            assert torch.equal(alone, whole[at:at + length]) and torch.equal(end[0], state[i])
        at += length


@pytest.mark.parametrize("d,dv", [(64, 64), (128, 128)])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.4028e38])
def test_a_value_stays_out_of_the_tokens_ahead_of_it(d, dv, value):
    n, at = 256, 122
    rows, before = inputs(n, d, dv, 1)
    clean, _ = step(rows, (n,), d, dv, before, torch.bfloat16)
    first_value, column = 2 * H * d, 5                                          # the first head's values
    rows[at, first_value + column] = value
    out, state = step(rows, (n,), d, dv, before, torch.bfloat16)
    assert torch.equal(out[:at // 16 * 16], clean[:at // 16 * 16])
    assert torch.equal(out[:, dv:], clean[:, dv:])                              # and out of the other heads
    others = [c for c in range(dv) if c != column]
    assert bool(torch.isfinite(state[0, 0][:, others]).all())                   # and out of the state's other columns
    if value < float("inf"):
        # the first head's decay, 0.4, has made the largest number an ordinary one by the end
        assert bool(torch.isfinite(state).all())


@pytest.mark.parametrize("d,dv", [(64, 64), (128, 128), (64, 128), (128, 64)])
@pytest.mark.parametrize("lengths", [(32,), (33, 31), (65, 127, 96), (128,), (129, 40), (384, 2, 300)])
def test_portions_of_many_heads_against_the_recurrence(d, dv, lengths):
    n = sum(lengths)
    rows, before = inputs(n, d, dv, len(lengths))
    results = {dtype: step(rows, lengths, d, dv, before, dtype) for dtype in (torch.float32, torch.bfloat16)}
    decay = torch.tensor([0.4, 0.97, 1 - 2.0 ** -9, 1.0] * (H // 4), device="cuda").double()
    q, k, v, gate = rows.double().split([H * d, H * d, H * dv, H * dv], dim=1)
    q, k, v = q.view(n, H, d), k.view(n, H, d), v.view(n, H, dv)
    want, end, at = torch.empty(n, H, dv, device="cuda", dtype=torch.float64), before.double(), 0
    for i, length in enumerate(lengths):
        for t in range(at, at + length):
            end[i] = decay[:, None, None] * end[i] + k[t][:, :, None] * v[t][:, None, :]
            want[t] = (end[i] * q[t][:, :, None]).sum(dim=1)
        at += length
    want = (want / torch.sqrt((want * want).mean(dim=-1, keepdim=True) + 1e-5)).view(n, H * dv) * gate * torch.sigmoid(gate)
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())
    # sums of up to 128 products at a time and of the chunks', their decays by exp2 of a 32-bit number: a few roundings of 2^-24, the outputs' also the
    # norm's and the gate's; then bfloat16's own
    assert rel(results[torch.float32][1], end) <= 4 * 2.0 ** -24 and rel(results[torch.float32][0], want) <= 12 * 2.0 ** -24
    assert rel(results[torch.bfloat16][0], want) <= 2.0 ** -9
