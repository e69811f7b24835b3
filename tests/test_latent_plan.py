"""How a step's prompt portions attend through a latent, decided on the host: what a captured step is replayed for."""
from types import SimpleNamespace

from lia_rs_b200.models.decoder import DecoderModel
from lia_rs_b200.parts.softmax_attention import LatentAttention


def layer(window):
    part = LatentAttention.__new__(LatentAttention)
    part.window, part.per_tile, part.heads, part.d, part.dr, part.dv, part.rank = window, 128, 16, 128, 64, 128, 512
    return part


def step(start, count=2048, page_size=16):
    cache = SimpleNamespace(page_size=page_size)
    return SimpleNamespace(n_tokens=count, n_out=1, context_bucket=4096, n_single=0, n_prefill_segments=1,
                           segments=[(0, start, count, 0)], runtime=SimpleNamespace(cache=cache))


def test_steps_of_one_graph_key_have_the_same_plans():
    layers = [layer(None), layer(128), layer(256)]
    model = SimpleNamespace(_key_layers=layers)
    plans = {}
    for start in list(range(200, 400)) + list(range(0, 40000, 97)):
        ctx = step(start)
        plan = [part._expansion(ctx) for part in layers]
        assert plans.setdefault(DecoderModel.graph_key(model, ctx), plan) == plan, start


def test_few_tokens_over_many_keys_stay_in_the_latents_space():
    wide, narrow = layer(None), layer(None)
    narrow.d, narrow.dr, narrow.dv, narrow.rank = 64, 32, 64, 256
    plans = lambda part, start, count: part._expansion(step(start, count)) is not None
    for part in (wide, narrow):
        assert not plans(part, 0, 15) and plans(part, 0, 16) and plans(part, 2000, 16) and plans(part, 30000, 32)
    assert not plans(wide, 8192, 20) and plans(wide, 8192, 21) and plans(narrow, 8192, 16)
    assert plans(layer(1024), 8192, 16)                                 # a window: the portion sees 1,039 keys


def test_the_expansion_keeps_to_its_memory():
    """Pages of 16 keys, 16 heads of 128 + 64 + 128 elements of two bytes: 6,553 pages fit into 1 GB, after rounding 6,144."""
    part = layer(None)
    assert part._expansion(step(6144 * 16 - 2048))[0] == 6144
    assert part._expansion(step(6144 * 16 - 2047)) is None


def test_the_profile_counts_what_the_path_computes(monkeypatch):
    from lia_rs_b200.kernels import ops
    monkeypatch.setattr(ops, "_profiler", object())
    part, ctx = layer(None), step(0, 100)
    pairs = 100 * 101 // 2
    assert part._work(ctx)[1] == 2 * 16 * (2 * 512 + 64) * pairs
    assert part._work(ctx, expanded=True)[1] == 2 * 16 * (128 + 64 + 128) * pairs
