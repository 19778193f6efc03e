"""Kevelorn without a GPU: the configuration's round trip and errors, the plan, the tensors the parts expect against an
independent list, what the cache is asked for, and the plain implementation's mechanisms on cases worked out by hand."""
from __future__ import annotations

import copy
import math
from types import SimpleNamespace

import pytest
import torch

import plain_kevelorn as plain
from kevelorn_models import CONFIGS, RANKS, make_weights, tensor_shapes


def build(name):
    from pico_engine.config.kevelorn import KevelornConfig
    from pico_engine.parts.model import DecoderModel
    cfg = CONFIGS[name]
    c = KevelornConfig.from_dict(cfg, tensor_shapes(cfg, RANKS[name]))
    return c, DecoderModel(c.plan(), torch.float32, "meta")


@pytest.mark.parametrize("name", sorted(CONFIGS))
def test_round_trip_and_expected_tensors(name):
    from pico_engine.config.registry import config_from_dict
    c, model = build(name)
    again = type(c).from_dict(c.to_dict())
    assert again.to_dict() == c.to_dict()
    assert type(config_from_dict(CONFIGS[name])) is type(c)
    expected = {n: tuple(s.shape) for n, s in model.expected_tensors().items()}
    assert expected == {n: tuple(s) for n, s in tensor_shapes(CONFIGS[name], RANKS[name]).items()}


def test_rank_comes_from_the_stored_tensor(tmp_path):
    from conftest import write_model
    from pico_engine.config.registry import read_config
    cfg = CONFIGS["K2"]
    folder = write_model(tmp_path / "m", cfg, make_weights(cfg, 0, RANKS["K2"]))
    assert read_config(folder).layers[0].decay_rank == RANKS["K2"]


def test_schedule_of_a_loop():
    c, model = build("K1")
    sched = model.plan.schedule
    assert [e.layer for e in sched] == [0, 1, 0, 1, 0, 1, 2]
    assert [e.add_vector for e in sched] == [("loop.step", 0), None, ("loop.step", 1), None, ("loop.step", 2), None, None]
    assert [e.add_embedding for e in sched] == [False, False, True, False, True, False, False]
    assert all(e.cache_of is None for e in sched)                      # every pass keeps its own keys, values and states
    c, model = build("K2")
    assert [e.layer for e in model.plan.schedule] == [0, 1, 2] and not model.plan.stream_vectors
    c, model = build("K4")
    assert [e.layer for e in model.plan.schedule] == [0, 1, 1]


def test_cache_needs():
    c, model = build("K1")
    needs = model.cache_needs()
    left = CONFIGS["K1"]["layers"][0]["mixer"]
    assert needs[0].kv.window == 40 and needs[0].kv.n_kv_heads == 2 and needs[0].kv.head_dim == 32
    assert needs[0].state_elems == 2 * 16 * 24 and needs[1].state_elems == 3 * 24 * 16 and needs[1].kv is None
    assert needs[6].state_elems == 3 * 40 * 8
    c, model = build("K2")
    assert model.cache_needs()[1].kv.value_shape == (4, 40) and model.cache_needs()[1].kv.window == 70
    c, model = build("K3")
    assert model.cache_needs()[1].kv.window is None


@pytest.mark.parametrize("change,word", [
    (lambda d: d["layers"][0].__setitem__("type", "conv"), "type"),
    (lambda d: d["layers"][0]["mixer"]["left"].__setitem__("kv_heads", 4), "evenly"),
    (lambda d: d["layers"][2]["mixer"].__setitem__("decay", [0.5]), "decay"),
    (lambda d: d["layers"][0]["mlp"]["router"].__setitem__("top", 9), "top"),
    (lambda d: d["loop"].__setitem__("stop", 7), "loop"),
    (lambda d: d["layers"][0]["mixer"]["left"]["rot"].__setitem__("dims", 34), "rot.dims"),
    (lambda d: d.pop("norm"), "norm"),
])
def test_errors_name_the_key(change, word):
    from pico_engine.config.kevelorn import KevelornConfig
    from pico_engine.config.specs import ConfigError
    d = copy.deepcopy(CONFIGS["K1"])
    change(d)
    with pytest.raises(ConfigError, match=word):
        KevelornConfig.from_dict(d)


# ------------------------------------------------------------------ the plain implementation on cases worked by hand

def test_rotation_by_hand():
    u = torch.zeros(3, 1, 6, dtype=torch.float64)
    u[:, 0] = torch.tensor([1.0, 0.0, 0.0, 2.0, 5.0, 7.0])
    out = plain.rotate_pairs(u, 2, 4, 100.0, 2.0)              # pairs (0,1), (2,3) turn; entries 4, 5 stay
    for t in range(3):
        p = 2 + t
        a0, a1 = p * 1.0 / 2.0, p * 100.0 ** -0.5 / 2.0
        assert torch.allclose(out[t, 0], torch.tensor([math.cos(a0), math.sin(a0), -2 * math.sin(a1), 2 * math.cos(a1), 5.0, 7.0], dtype=torch.float64))


def test_window_by_hand():
    n = 6
    q = torch.zeros(n, 2, 2, dtype=torch.float64)
    k = torch.zeros(n, 1, 2, dtype=torch.float64)
    v = torch.arange(n, dtype=torch.float64).view(n, 1, 1)
    out = plain.window_attention(q, k, v, 1.0, 3)              # equal scores: the mean of the visible values
    assert torch.allclose(out[:, 0, 0], torch.tensor([0.0, 0.5, 1.0, 2.0, 3.0, 4.0], dtype=torch.float64))
    assert torch.allclose(plain.window_attention(q, k, v, 1.0, 1)[:, 1, 0], v.view(-1))
    assert torch.allclose(plain.window_attention(q, k, v, 1.0, None)[:, 0, 0], torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 2.5], dtype=torch.float64))


def test_recurrence_by_hand():
    q = torch.ones(3, 1, 1, dtype=torch.float64)
    k = torch.ones(3, 1, 1, dtype=torch.float64)
    v = torch.tensor([1.0, 10.0, 100.0], dtype=torch.float64).view(3, 1, 1)
    o, S = plain.linear_recurrence(q, k, v, torch.full((3, 1, 1), 0.5, dtype=torch.float64))
    assert o.view(-1).tolist() == [1.0, 10.5, 105.25] and float(S) == 105.25
    o2, _ = plain.linear_recurrence(q[2:], k[2:], v[2:], torch.full((1, 1, 1), 0.5, dtype=torch.float64), state=torch.tensor([[[10.5]]], dtype=torch.float64))
    assert float(o2) == 105.25


def test_mixture_by_hand():
    W = 2
    w = {"r.router": torch.tensor([[1.0, 0.0], [0.0, 1.0], [-1.0, -1.0]], dtype=torch.float64)}
    for e in range(3):
        w[f"r.e{e}.gate"] = torch.full((1, W), 50.0, dtype=torch.float64)       # silu(large) = itself
        w[f"r.e{e}.up"] = torch.full((1, W), float(e + 1), dtype=torch.float64)
        w[f"r.e{e}.down"] = torch.ones(W, 1, dtype=torch.float64)
    h = torch.tensor([[2.0, 1.0]], dtype=torch.float64)
    out = plain.mixture(h, w, "r.", {"router": {"experts": 3, "top": 2}})
    p0 = math.exp(2) / (math.exp(2) + math.exp(1))
    gate = 150.0                                                                 # 50 * (2 + 1)
    assert torch.allclose(out, torch.full((1, W), gate * (p0 * 3.0 + (1 - p0) * 6.0), dtype=torch.float64))


def test_layer_runs():
    assert plain.layer_runs({"layers": [0] * 4, "loop": {"start": 1, "stop": 3, "times": 2}}) == \
        [(0, None), (1, 0), (2, None), (1, 1), (2, None), (3, None)]
    assert plain.layer_runs({"layers": [0] * 2}) == [(0, None), (1, None)]


@pytest.mark.parametrize("per_channel", [0, 1])
def test_scratch_of_a_batch_of_prompts_is_bounded(per_channel):
    """A recurrence in chunks takes a batch's chunks in slabs: 64 prompts of 2,048 tokens need no more scratch than a few prompts do."""
    from pico_engine.ops.library import gated, state_space
    for H, D in ((16, 128), (32, 128), (14, 64), (3, 250)):
        one, many = (gated().pe_linear_attention_scratch_floats(2048 * n, n, H, D, D, per_channel) for n in (1, 64))
        assert 0 < 4 * one <= 256 << 20 and 4 * many <= 256 << 20
        assert gated().pe_linear_attention_slabs(2048, 1, H, D, D, per_channel) == 1 < gated().pe_linear_attention_slabs(2048 * 64, 64, H, D, D, per_channel)
    assert 4 * state_space().pe_state_space_scratch_floats(2048 * 64, 64, 64, 64, 128, 2) <= 256 << 20
    assert state_space().pe_state_space_slabs(2048, 1, 64, 64, 128, 2) == 1


@pytest.mark.parametrize("per_channel", [0, 1])
def test_scratch_is_what_the_way_of_a_step_takes(per_channel):
    """Float32 rows have no parts and rows without an activation on the values none of those: neither pays for them with smaller slabs."""
    from pico_engine.ops.library import gated
    lib, H, D = gated(), 16, 128
    adds, parts, values = (lib.pe_linear_attention_scratch_floats(200, 1, H, D, D, per_channel | kind) - 8 for kind in (0, 2, 6))
    state = 5 * H * D * (D + 1)
    assert adds == state + per_channel * 5 * H * (64 * 64 + 2 * 64 * D)
    assert parts == state + 5 * (H * 15 * 8192 // 4 + 2 * H + 2) and values - parts == 5 * H * 6 * 8192 // 4
    T = 64 * (253 if per_channel == 0 else 108)
    assert [lib.pe_linear_attention_slabs(T, 1, H, D, D, per_channel | kind) for kind in (0, 2, 6)] == ([1, 3, 4] if per_channel == 0 else [1, 2, 2])


@pytest.mark.parametrize("values", [0, 4])
@pytest.mark.parametrize("per_channel", [0, 1])
@pytest.mark.parametrize("D", [64, 128])
def test_scratch_of_the_tensor_cores_is_aligned_for_what_reads_it(D, per_channel, values):
    """Any number of heads and chunks, odd ones too: parts and states start where 16 and 32 bytes are read at once, a chunk's place where 8 are,
    nothing overlaps and all of it lies in the scratch."""
    import ctypes
    from pico_engine.ops.library import gated
    lib, places = gated(), (ctypes.c_longlong * 5)()
    for H in range(1, 17):
        for chunks in range(2, 200):
            T = 64 * (chunks - 1)
            sizes = (T, 1, H, D, D, per_channel | 2 | values)
            if not lib.pe_linear_attention_scratch_places(*sizes, ctypes.addressof(places)):
                assert D == 64 and H % 2
                continue
            rows, seen, state, decay, end = places
            slab = -(-chunks // lib.pe_linear_attention_slabs(*sizes))
            assert rows % 16 == 0 and seen % 4 == 0 and state % 32 == 0 and decay % 16 == 0, (H, chunks)
            planes = (12 + 3 * (1 if D == 128 else 2) + (6 if values else 0)) * 8192 * (H if D == 128 else H // 2)
            assert rows >= slab * planes and seen - rows >= 8 * slab and state - seen >= 8 * slab * H and decay - state >= 4 * slab * H * D * D
            assert end - decay >= 4 * slab * H * D and end <= 4 * lib.pe_linear_attention_scratch_floats(*sizes), (H, chunks)


ONES = [1] * 63


@pytest.mark.parametrize("per_channel,heads,dim,walks,chunks", [
    (True, 16, 128, [[17], [64], [96], [10, 64, 54], [17] * 64, [64] * 64, [128] * 16, [200] + ONES], [[256], [512], [2048], [512] * 4, [2048] + ONES]),
    (True, 14, 64, [[17], [64], [17] * 64, [128] * 64, [200] + ONES], [[256], [2048], [512] * 4, [2048] + ONES]),
    (False, 16, 128, [[17], [64], [17] * 64, [64] * 64, [200] + ONES], [[256], [512], [2048], [512] * 4, [2048] + ONES]),
    (False, 14, 64, [[17], [64], [17] * 64, [128] * 64, [200] + ONES], [[256], [2048], [512] * 4, [2048] + ONES])])
def test_linear_attention_takes_the_way_that_was_measured_shorter(per_channel, heads, dim, walks, chunks):
    """Steps whose two ways differed by a fifth and more on a B200 (tokens a row): from one row to 64, short and long, equal and not."""
    from pico_engine.parts.linear_attention import LinearAttention
    part = SimpleNamespace(spec=SimpleNamespace(n_heads=heads, head_dim=dim, v_head_dim=dim), head_decay=None if per_channel else object())
    for way, steps in ((False, walks + [[1], [16], [1] * 64]), (True, chunks)):
        for lens in steps:
            assert LinearAttention.chunks_pay(part, lens) == way, lens


@pytest.mark.parametrize("heads,state,walks,chunks", [
    (64, 128, [[17], [24], [17] * 8, [24] * 64, [200] + ONES], [[96], [2048], [64] * 8, [128] * 64, [2048] + ONES]),
    (28, 128, [[17], [24], [17] * 8, [24] * 64, [200] + ONES], [[64], [2048], [64] * 8, [128] * 64, [2048] + ONES]),
    (16, 64, [[17], [17] * 16, [24] * 64], [[64], [2048], [96] * 8, [256] * 64, [2048] + ONES])])
def test_state_space_takes_the_way_that_was_measured_shorter(heads, state, walks, chunks):
    """The same for the state-space recurrence, 64 columns a head."""
    from pico_engine.parts.state_space import StateSpace
    part = SimpleNamespace(spec=SimpleNamespace(n_heads=heads, head_dim=64, state=state))
    for way, steps in ((False, walks + [[1], [16], [1] * 64]), (True, chunks)):
        for lens in steps:
            assert StateSpace.chunks_pay(part, lens) == way, lens

