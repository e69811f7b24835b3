"""Retention's prompt portions in tiles (heads of 64 or 128 elements) against the plain recurrence in 64-bit, and beside the kernels
for every size: portions around the chunks' and the warps' edges, several at once, continuing from states of their own."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def plain(rows, decay, before, H, d, dv, eps):
    q, k, v, g = (x.to(F64) for x in rows.split([H * d, H * d, H * dv, H * dv], dim=1))
    n = rows.shape[0]
    q, k, v = q.view(n, H, d), k.view(n, H, d), v.view(n, H, dv)
    S, out = before.to(F64).clone(), torch.zeros(n, H, dv, dtype=F64, device=rows.device)
    for t in range(n):
        S = decay.to(F64)[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
        out[t] = (S * q[t][:, :, None]).sum(dim=1)
    out = out / torch.sqrt((out * out).mean(dim=-1, keepdim=True) + eps)
    return out.reshape(n, H * dv) * g * torch.sigmoid(g), S


@pytest.mark.parametrize("d,dv", [(64, 64), (64, 128), (128, 64), (128, 128)])
@pytest.mark.parametrize("lengths", [(2,), (15, 16), (17, 63), (64, 2, 65), (130, 129)])
def test_tiles_against_the_plain_recurrence(d, dv, lengths):
    from lia_rs_b200.kernels import ops
    gen = torch.Generator(device="cuda").manual_seed(d + dv + len(lengths))
    H, eps, n = 3, 1e-5, sum(lengths)
    width = 2 * H * (d + dv)
    rows = torch.randn(n, width, device="cuda", generator=gen)
    rows[:, H * d:2 * H * d] *= d ** -0.5
    decay = torch.tensor([1.0, 0.97, 0.4], device="cuda")
    before = torch.randn(5, H, d, dv, device="cuda", generator=gen)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    slots_of = [4, 0, 2][:len(lengths)]
    segments, slots, want, ends, at = [], [], [], before.to(F64).clone(), 0
    for slot, count in zip(slots_of, lengths):
        segments += [at, 7, count]
        slots += [slot] * count
        out, ends[slot] = plain(rows[at:at + count], decay, before[slot], H, d, dv, eps)
        want.append(out)
        at += count
    want = torch.cat(want)
    chunks = ops.retention_chunks(n, len(lengths))
    scratch = torch.empty(ops.retention_scratch_floats(chunks, H, d, dv), device="cuda")

    def run(rows, dtype=torch.float32):
        state, out = before.clone(), torch.zeros(n, H * dv, dtype=dtype, device="cuda")
        ops.retention(rows, decay, state, ints(segments), len(lengths), chunks, ints([]), ints(slots), out, H, d, dv, eps, scratch=scratch)
        return out, state

    out, state = run(rows)
    crooked = torch.zeros(n, width + 1, device="cuda")              # rows that no 16-byte load can read: the kernels for every size
    crooked[:, :width] = rows
    other, other_state = run(crooked)
    off = lambda a, b: float((a.to(F64) - b).norm() / b.norm())
    # the same sums in another order: at most twice as far from 64 bits as the kernels for every size, or within a few roundings
    assert off(out, want) < 2 * off(other, want) + 2.0 ** -22, (off(out, want), off(other, want))
    assert off(state, ends) < 2 * off(other_state, ends) + 2.0 ** -22, (off(state, ends), off(other_state, ends))
    assert off(out, want) < 1e-5 and off(state, ends) < 2e-6
    rounded, _ = run(rows, torch.bfloat16)
    assert torch.equal(rounded, out.to(torch.bfloat16))
