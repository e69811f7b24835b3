"""Attention through a latent whose prompt portions are expanded into whole keys and values: portions around the tiles' and
pages' edges, late in their prompts, windows, gates, and single tokens in the same step, against the plain functions in 64-bit."""
import pytest
import torch

import plain_vatunex as pv
import plain_zipelix as pz
from test_botuvik_parts_gpu import PartRunner

pytestmark = pytest.mark.gpu
F64 = torch.float64
# eight values are rounded to bfloat16 on the way (queries, latents, keys, values, probabilities, outputs and the two products'
# operands), each by at most 2^-8 of itself and by less than 2^-9 in the root mean square (a uniform error over the numbers between
# two powers of two: 0.41 * 2^-8), and the result is linear in each: 8 * 2^-9 of its size in the Euclidean norm, if all add up
REL = 8 * 2.0 ** -9


def tensors(hidden, m, form, g):
    H, d, dr, dv, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    shapes = {"dkv": (rank + dr, hidden), "uk": (H * d, rank), "uv": (H * dv, rank), "o": (hidden, H * dv)}
    if form == "windowed":
        shapes.update({"dq": (64, hidden), "uq": (H * (d + dr), 64)})
    else:
        shapes.update({"q": (H * (d + dr), hidden), "g": (H * dv, hidden)})
    w = {name: (torch.randn(*shape, generator=g) * shape[1] ** -0.5).to(torch.bfloat16) for name, shape in shapes.items()}
    w["dkv.norm"] = (1 + 0.1 * torch.randn(rank, generator=g)).to(torch.bfloat16)
    if form == "windowed":
        w["dq.norm"] = (1 + 0.1 * torch.randn(64, generator=g)).to(torch.bfloat16)
    return w


@pytest.mark.parametrize("d,dr,dv,rank,page", [(128, 64, 128, 512, 16), (64, 32, 64, 256, 16), (64, 64, 64, 32, 5), (32, 32, 128, 96, 8)])
@pytest.mark.parametrize("form", ["gated", "windowed"])
def test_expanded_portions_against_plain_functions(d, dr, dv, rank, page, form):
    g = torch.Generator().manual_seed(d + rank)
    hidden, heads = 96, 3
    m = dict(heads=heads, dim=d, rot_dim=dr, vdim=dv, kv_rank=rank, scale=(d + dr) ** -0.5, rot={"base": 100.0, "dims": dr})
    if form == "windowed":
        m["mask"] = {"size": 70}
    w = tensors(hidden, m, form, g)
    params = dict(hidden=hidden, heads=heads, head_dim=d, rot_dim=dr, v_head_dim=dv, kv_rank=rank, scale=m["scale"], norm_eps=1e-5,
                  rot=m["rot"], **(dict(q_rank=None, gate="sigmoid", rot_pairs=True) if form == "gated" else
                                   dict(q_rank=64, window=70)))
    runner = PartRunner("latent_attention", params, w, "bfloat16", page_size=page, slots=4, tokens=1024)
    part = runner.part
    assert part.per_tile == 128
    lengths = {"a": 420, "b": 257, "c": 140, "e": 40}
    rows = {name: torch.randn(n, hidden, generator=g).to(torch.bfloat16).float() for name, n in lengths.items()}
    # whole tiles and their neighbours, portions late in a prompt, single tokens beside portions and alone
    steps = [[("a", 128), ("b", 129)], [("a", 127), ("c", 17), ("b", 1)], [("a", 1), ("b", 1)], [("a", 2), ("b", 33), ("c", 121), ("e", 20)],
             [("a", 162), ("b", 1), ("e", 18), ("c", 1)], [("b", 92), ("c", 1), ("e", 2)]]
    got = {name: [] for name in lengths}
    for entries in steps:
        for name, out in runner.step(entries, rows).items():
            got[name].append(out)
    for name, length in lengths.items():
        h, positions = rows[name].to(F64), torch.arange(length)
        if form == "gated":
            cache = pz.latent_cache(h, positions, w["dkv"], w["dkv.norm"], m, 1e-5)
            want = pz.latent_attention(h, positions, w, m, cache)
        else:
            want = pv.latent_attention(m, lambda key: w[key].to(F64), h, positions, 1e-5)
        out = torch.cat(got[name])
        assert out.shape == want.shape
        assert float((out - want).norm() / want.norm()) < REL, (name, float((out - want).norm() / want.norm()))
        assert float((out - want).norm(dim=-1).max() / want.norm(dim=-1).max()) < 2 * REL


@pytest.mark.parametrize("page,pages", [(16, [7, 12]), (1, [104, 192])])
def test_a_prompt_that_outgrows_the_expansion(page, pages, monkeypatch):
    """Portions of one prompt on both sides of the expansion's memory limit: the same attention."""
    from lia_rs_b200.parts.softmax_attention import LatentAttention
    g = torch.Generator().manual_seed(9)
    m = dict(heads=3, dim=64, rot_dim=32, vdim=64, kv_rank=256, scale=96 ** -0.5, rot={"base": 100.0, "dims": 32})
    w = tensors(96, m, "gated", g)
    params = dict(hidden=96, heads=3, head_dim=64, rot_dim=32, v_head_dim=64, kv_rank=256, scale=m["scale"], norm_eps=1e-5,
                  rot=m["rot"], q_rank=None, gate="sigmoid", rot_pairs=True)
    runner = PartRunner("latent_attention", params, w, "bfloat16", page_size=page, slots=page, tokens=1024)
    monkeypatch.setattr(LatentAttention, "EXPAND_BYTES", 192 * 3 * 160 * 2)                      # 192 keys
    ways, rows, got = [], {"a": torch.randn(500, 96, generator=g).to(torch.bfloat16).float()}, []
    whole = LatentAttention._expansion
    monkeypatch.setattr(LatentAttention, "_expansion", lambda part, ctx: ways.append(whole(part, ctx)) or ways[-1])
    for count in (100, 92, 60, 248):
        got.append(runner.step([("a", count)], rows)["a"])
    assert [way and way[0] for way in ways] == pages + [None, None]
    h, positions = rows["a"].to(F64), torch.arange(500)
    want = pz.latent_attention(h, positions, w, m, pz.latent_cache(h, positions, w["dkv"], w["dkv.norm"], m, 1e-5))
    off = torch.cat(got) - want
    assert float(off.norm() / want.norm()) < REL and float(off.norm(dim=-1).max() / want.norm(dim=-1).max()) < 2 * REL


def test_which_portions_are_expanded():
    """The rule looks at the portions alone: long enough on average and not beyond the memory it may take; the pages it names
    cover what the portions see, rounded up by less than an eighth."""
    from types import SimpleNamespace
    params = dict(hidden=96, heads=2, head_dim=64, rot_dim=32, v_head_dim=64, kv_rank=32, scale=0.1, rot=None, q_rank=None)
    g = torch.Generator().manual_seed(1)
    m = dict(heads=2, dim=64, rot_dim=32, vdim=64, kv_rank=32)
    w = tensors(96, m, "gated", g)
    w.pop("g")
    part = PartRunner("latent_attention", params, w, "bfloat16", page_size=16, slots=2, tokens=64).part

    def plan(segments, page_size=16):
        portions = sum(1 for _, _, count, _ in segments if count > 1)
        return part._expansion(SimpleNamespace(n_prefill_segments=portions, segments=segments,
                                               runtime=SimpleNamespace(cache=SimpleNamespace(page_size=page_size))))

    assert plan([(0, 5, 1, 0)]) is None
    assert plan([(0, 0, 15, 0)]) is None and plan([(0, 0, 16, 0)]) == (1, 1)
    assert plan([(0, 0, 2048, 0), (1, 7, 1, 2048)]) == (128, 16)
    for last in range(17, 3000, 41):
        pages, tiles = plan([(0, last - 17, 17, 0), (1, 0, 130, 17)])
        seen = (last + 15) // 16 + 9
        assert seen <= pages < seen * 9 / 8 + 1 and tiles == 3
    assert plan([(0, 1 << 24, 64, 0)]) is None


def test_contiguous_tensors_of_any_shape_and_stride():
    """Contiguous outputs of latent_prepare in other shapes, and dimensions of size one with strides that mean nothing."""
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(2)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    H, d, dr, rank, page = 3, 32, 16, 32, 4
    odd = lambda t, dim: t.as_strided(t.shape, [0 if i == dim else s for i, s in enumerate(t.stride())], t.storage_offset())

    def prepare(n, plain, rotated):
        rows = torch.randn(n, H * (d + dr), device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
        pages = [torch.zeros(4, page, 1, size, device="cuda", dtype=torch.bfloat16) for size in (rank, dr)]
        freq = torch.full((dr // 2,), 0.3, device="cuda")
        ops.latent_prepare(rows, None, None, 1e-5, freq, dr, ints(list(range(n))), ints([0] * n), ints([[0, 1, 2, 3]]), plain, rotated,
                           *pages, H, d, dr, rank)
        return plain.reshape(-1), rotated.reshape(-1)

    zeros = lambda *shape: torch.zeros(*shape, device="cuda", dtype=torch.bfloat16)
    want = prepare(5, zeros(H, 5, d), zeros(5, H * dr))
    assert float(want[0].float().abs().sum()) > 0 < float(want[1].float().abs().sum())
    for plain, rotated in ((zeros(H * 5, d), zeros(5 * H, dr)), (zeros(H * 5 * d), zeros(5, H, dr)), (zeros(5, H * d), zeros(5 * H * dr))):
        got = prepare(5, plain, rotated)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    want = prepare(1, zeros(H, 1, d), zeros(1, H * dr))
    got = prepare(1, odd(zeros(H, 1, d), 1), odd(zeros(1, H * dr), 0))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])

    x, weight = torch.randn(1, 64, device="cuda", generator=g), torch.ones(64, device="cuda")
    out, other = (torch.zeros(1, 64, device="cuda") for _ in range(2))
    ops.rmsnorm(x, weight, out, 1e-5)
    ops.rmsnorm(odd(x, 0), weight, other, 1e-5)
    assert torch.equal(out, other) and float(out.abs().sum()) > 0

    q = torch.randn(9, 2 * 64, device="cuda", generator=g).to(torch.bfloat16)
    k, v = (torch.randn(1, 16, 1, 64, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    results = []
    for keys, values in ((k, v), (odd(k, 0), odd(v, 2)), (k[:, :, 0], v[:, :, 0])):
        out = torch.zeros_like(q)
        ops.attention_prefill_tc(q, keys, values, ints([0, 0, 9]), 1, 1, ints([0] * 9), ints([[0]]), out, 2, 1, 64, None, 0.1)
        results.append(out)
    assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2]) and float(out.float().abs().sum()) > 0


@pytest.mark.parametrize("d,dv", [(192, 128), (96, 64)])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("form", ["none", "elements", "unaligned elements", "heads"])
def test_gated_epilogue_against_64_bits(d, dv, splits, form):
    """Whole keys and values of an expanded latent, the keys whole or in ranges, the output times the gate's sigmoid."""
    from lia_rs_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(d + splits)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    H, page, portions = 3, 8, [(1, 300, 150), (0, 0, 2), (2, 120, 129)]              # slot, first position, tokens
    n, blocks = sum(p[2] for p in portions), 60
    q = torch.randn(n, H * d, device="cuda", generator=g).to(torch.bfloat16)
    rows = torch.randn(3 * blocks, page, H * (d + dv), device="cuda", generator=g).to(torch.bfloat16)       # keys of all heads, then values
    keys, values = rows[:, :, :H * d].unflatten(2, (H, d)), rows[:, :, H * d:].unflatten(2, (H, dv))
    table = torch.randperm(3 * blocks, generator=torch.Generator().manual_seed(1)).view(3, blocks).to(torch.int32).cuda()
    first = 3 if form == "unaligned elements" else 4                                 # the gate's columns behind others
    gate = None if form == "none" else 4 * torch.randn(n, first + H * dv, device="cuda", generator=g)[:, first:]
    if form == "heads":
        gate = gate[:, :H]
    segments, slots, want, at = [], [], [], 0
    for slot, start, count in portions:
        segments += [at, start, count]
        slots += [slot] * count
        mine = rows[table[slot].long()].reshape(blocks * page, -1)[:start + count].double()
        k, v = mine[:, :H * d].view(-1, H, d), mine[:, H * d:].view(-1, H, dv)
        scores = torch.einsum("thd,jhd->htj", q[at:at + count].double().view(count, H, d), k) * d ** -0.5
        later = torch.arange(start + count, device="cuda") > torch.arange(start, start + count, device="cuda")[:, None]
        want.append(torch.einsum("htj,jhv->thv", scores.masked_fill(later, float("-inf")).softmax(-1), v))
        at += count
    want = torch.cat(want)
    if gate is not None:
        want = want * torch.sigmoid(gate.double().reshape(n, H, -1))
    out, flag = torch.zeros(n, H * dv, device="cuda", dtype=torch.bfloat16), ints([0])
    tiles = sum((count + 127) // 128 for _, _, count in portions)
    partial = torch.empty(ops.attention_prefill_tc_partial_floats(n, H, dv, splits), device="cuda") if splits > 1 else None
    call = lambda gate: ops.attention_prefill_tc(q, keys, values, ints(segments), 3, tiles, ints(slots), table, out, H, H, d, None, d ** -0.5,
                                                 flag, splits=splits, partial=partial, gate=gate, gate_head=form == "heads")
    call(gate)
    # probabilities and outputs are rounded to 16 bits, 2^-9 of themselves each, and the output is linear in both
    off = (out.double().view(n, H, dv) - want).norm() / want.norm()
    assert float(off) < 2 * 2.0 ** -9 and int(flag) == 0
    if gate is not None:
        with pytest.raises(ops.KernelError):
            call(gate.cpu())
