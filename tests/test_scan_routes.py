"""Which kernel a selective scan's portions go to, by their sizes; and that what the caller sees does not depend on it."""
import pytest
import torch

from lia_rs_b200.kernels import ops


def walks(channels, states, tokens, portions=1, n_single=0):
    x = torch.empty(1).expand(tokens + n_single, channels)
    bc = torch.empty(1).expand(tokens + n_single, 2 * states)
    return ops.selective_scan_walks_runs(x, x, bc, 0, states, x, x, states, portions, n_single)


@pytest.mark.parametrize("states,channels,last", [(4, 256, 1280), (4, 1024, 2304), (8, 256, 2304), (16, 256, 2560), (16, 512, 4096), (64, 256, 1280)])
def test_long_portions_of_few_channels_are_cut(states, channels, last):
    assert walks(channels, states, last) and not walks(channels, states, 2 * last)
    assert walks(channels, states, 8 * last, 8)                          # as long each, side by side: the device is less idle
    assert walks(4096, 16, 8192) and walks(2048, 16, 8192)


def test_short_portions_go_with_the_single_tokens():
    assert walks(4096, 16, 2) and walks(256, 16, 21, 3)                  # nothing to share a launch with
    assert not walks(256, 16, 7, 1, 1) and walks(256, 16, 8, 1, 1)
    assert not walks(4096, 16, 31, 4) and walks(4096, 16, 32, 4)         # more CTAs than a round


@pytest.mark.gpu
@pytest.mark.parametrize("channels,states,lengths,n_single", [(32, 4, (1600,), 0), (64, 64, (1200,), 3), (64, 16, (2, 7, 3), 5), (8, 8, (2,), 1),
                                                              (8192, 4, (3, 4), 0)])
def test_portions_that_stay_with_the_kernels_for_every_size(channels, states, lengths, n_single):
    """The same bits as rows that the kernel for whole portions cannot read, which those kernels serve."""
    g = torch.Generator(device="cuda").manual_seed(channels + states)
    rnd = lambda *shape: torch.randn(*shape, device="cuda", generator=g)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    n = sum(lengths) + n_single
    x, dt_raw, bc, D, bias = rnd(n, channels), rnd(n, channels), rnd(n, 2 * states), rnd(channels), rnd(channels) - 1
    A, wide, before = -torch.exp(rnd(channels, states)), rnd(n, channels + 1), rnd(len(lengths) + n_single, channels, states)
    segments, slots, at = [], [], 0
    for slot, length in enumerate(lengths):
        segments += [at, 0, length]
        slots += [slot] * length
        at += length
    singles, slots = list(range(at, n)), slots + [len(lengths) + i for i in range(n_single)]
    results = []
    for z in (wide[:, :channels].contiguous(), wide[:, :channels]):
        out, state = torch.zeros(n, channels, device="cuda"), before.clone()
        assert not ops.selective_scan_walks_runs(x, dt_raw, bc, 0, states, z, out, states, len(lengths), n_single)
        scratch = torch.empty(ops.selective_scan_chunk_floats(n, len(lengths), channels, states), device="cuda") if n >= 256 else None
        ops.selective_scan(x, dt_raw, bias, A, bc, 0, states, D, z, state, ints(segments), len(lengths), ints(singles), ints(slots), out,
                           chunk_scratch=scratch)
        results.append((out, state))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    assert float(results[0][0].abs().min(dim=1).values.max()) > 0 and not torch.equal(results[0][1], before)
