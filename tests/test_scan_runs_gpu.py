"""The kernel that walks whole portions of a selective scan, sixteen lanes a channel, against the plain recurrence in 64-bit and the
kernel for every size; and the convolution that gives a thread eight rows, against the one that gives it one."""
import pytest
import torch

import plain_vatunex as pv

pytestmark = pytest.mark.gpu
F64 = torch.float64


def ints(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("channels,states", [(4, 4), (8, 8), (12, 12), (20, 16), (64, 16), (36, 20), (8, 32), (40, 64)])
@pytest.mark.parametrize("lengths", [(2,), (7, 8), (9, 31, 2), (32, 33), (70, 3, 64)])
def test_runs_against_the_plain_recurrence(channels, states, lengths):
    from lia_rs_b200.kernels import ops
    g = torch.Generator().manual_seed(channels * 100 + states + len(lengths))
    taps, rank = 4, 8
    n = sum(lengths)
    x, dt_raw = torch.randn(n, channels, generator=g), torch.randn(n, channels, generator=g)
    uz = torch.randn(n, 2 * channels, generator=g)
    projected = torch.randn(n, rank + 2 * states, generator=g)
    A = -torch.exp(torch.randn(channels, states, generator=g))
    D, bias = torch.randn(channels, generator=g), torch.randn(channels, generator=g) - 1
    before = torch.randn(4, channels, states, generator=g)
    inputs = torch.randn(4, taps - 1, channels, generator=g)
    slots_of, starts = [2, 0, 3][:len(lengths)], [5, 0, 40][:len(lengths)]
    segments, slots, positions, at = [], [], [], 0
    for slot, start, length in zip(slots_of, starts, lengths):
        segments += [at, start, length]
        slots += [slot] * length
        positions += list(range(start, start + length))
        at += length
    want, end = torch.zeros(n, channels, dtype=F64), before.to(F64).clone()
    z = uz[:, channels:].to(F64)
    for i, slot in enumerate(slots_of):
        first, length = segments[3 * i], lengths[i]
        S = before[slot].to(F64)
        for t in range(first, first + length):
            dt = torch.nn.functional.softplus(dt_raw[t].to(F64) + bias)
            S = torch.exp(dt[:, None] * A) * S + (dt * x[t])[:, None] * projected[t, rank:rank + states].to(F64)
            want[t] = (S @ projected[t, rank + states:].to(F64) + D * x[t]) * z[t] * torch.sigmoid(z[t])
        end[slot] = S
    dev = lambda t: t.cuda()
    args = (dev(x), dev(dt_raw), dev(bias), dev(A), dev(projected), rank, rank + states, dev(D))
    state, conv_state, wide = dev(before.clone()), dev(inputs.clone()), dev(uz)
    out = torch.zeros(n, channels, device="cuda")
    assert ops.selective_scan_walks_runs(args[0], args[1], args[4], rank, rank + states, wide[:, channels:], out, states)
    ops.selective_scan(*args, wide[:, channels:], state, ints(segments), len(lengths), ints([]), ints(slots), out,
                       conv_state=conv_state, conv_x=wide)
    # 32-bit sums of at most 70 decayed terms and 64 products: the errors stay below 2^-24 times their number times the largest term
    scale = float(want.abs().max())
    assert float((out.cpu().to(F64) - want).abs().max()) < 70 * 2.0 ** -24 * 8 * scale
    assert float((state.cpu().to(F64) - end).abs().max()) < 70 * 2.0 ** -24 * 4 * float(end.abs().max())
    # the convolution's state, as the kernel of its own leaves it
    reference = dev(inputs.clone())
    ops.conv_state_update(wide, reference, ints(positions), ints(slots), channels)
    assert torch.equal(conv_state, reference)
    # the kernel for every size (rows of z that no 16-byte load can read)
    crooked = torch.zeros(n, channels + 1, device="cuda")
    crooked[:, :channels] = wide[:, channels:]
    assert not ops.selective_scan_walks_runs(args[0], args[1], args[4], rank, rank + states, crooked[:, :channels], out, states)
    other, other_state = torch.zeros_like(out), dev(before.clone())
    ops.selective_scan(*args, crooked[:, :channels], other_state, ints(segments), len(lengths), ints([]), ints(slots), other)
    assert torch.allclose(out, other, atol=2e-5 * scale, rtol=2e-5)
    rounded = torch.zeros(n, channels, dtype=torch.bfloat16, device="cuda")
    ops.selective_scan(*args, wide[:, channels:], dev(before.clone()), ints(segments), len(lengths), ints([]), ints(slots), rounded)
    assert torch.equal(rounded, out.to(torch.bfloat16))


@pytest.mark.parametrize("taps", [2, 3, 4, 6])
@pytest.mark.parametrize("channels", [4, 36, 516, 3324])
def test_convolution_of_eight_rows_a_thread(taps, channels):
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(taps * 1000 + channels)
    rnd = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    # runs that begin and end inside a tile, single tokens, a row of nobody, a sequence's start
    runs = [(1, 40, 20), (0, 0, 1), (3, 7, 1), (2, 1, 30), (4, 0, 65), (5, 2, 2)]
    slots = [s for s, _, n in runs for _ in range(n)] + [-1] * 3
    positions = [p for _, first, n in runs for p in range(first, first + n)] + [0] * 3
    n = len(slots)
    x, w, b, state = rnd(n, 2 * channels), rnd(channels, taps), rnd(channels), rnd(6, taps - 1, channels)
    results = []
    for rows in (x, torch.cat([x, x[:, :1]], dim=1)[:, :2 * channels]):          # the second: rows no 16-byte load can read
        out, copy = torch.zeros(n, channels, device="cuda"), torch.zeros(n, channels, dtype=torch.bfloat16, device="cuda")
        ops.causal_conv(rows, w, b, state, ints(positions), ints(slots), out, copy, act=1)
        results.append((out, copy))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    assert torch.equal(results[0][1], results[0][0].to(torch.bfloat16)) and float(results[0][0][-3:].abs().max()) == 0.0
