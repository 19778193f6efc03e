"""Kevelorn on the GPU against the plain implementation: each mechanism's kernel alone on inputs that show a fault,
and the whole model through the library's step function, cache, scheduler and entry points, in both dtypes, for
every way of cutting requests into steps."""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import pytest
import torch

import plain_kevelorn as plain
import replay
from conftest import write_model
from kevelorn_models import CONFIGS, RANKS, make_weights, plain_logits, requests_for

pytestmark = pytest.mark.gpu

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}
CASES = [(n, d) for n in sorted(CONFIGS) for d in ("float32", "bfloat16")]
LENGTHS = {"K1": [1, 2, 3, 37, 70, 131, 64, 5], "K2": [65, 1, 150, 9, 33, 2], "K3": [3, 129, 31, 64, 1, 200], "K4": [4, 1, 90, 17, 66]}


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    """{(config, dtype): (engine, cfg, weights, folder)}."""
    from pico_engine.engine.engine import Engine
    root = tmp_path_factory.mktemp("kevelorn")
    out = {}
    for k, (name, cfg) in enumerate(sorted(CONFIGS.items())):
        weights = make_weights(cfg, 40 + k, RANKS[name])
        folder = write_model(root / name, cfg, weights)
        for dtype in DTYPES:
            out[(name, dtype)] = (Engine(folder, dtype=dtype), cfg, weights, folder)
    return out


def compare(got, cfg, w, reqs, dtype, what, only_got=False):
    """Against the plain logits; in bfloat16 without the places where the plain router's choice was a close call."""
    close = set()
    want = plain_logits(cfg, w, reqs, close)
    if only_got:
        want = {k: v for k, v in want.items() if k in got}
    if dtype == "bfloat16":
        assert len(close) < 0.5 * len(want)
        got, want = ({k: v for k, v in d.items() if k not in close} for d in (got, want))
    replay.compare(got, want, dtype, what)


def check(models, name, dtype, steps, reqs, what):
    eng, cfg, w, _ = models[(name, dtype)]
    compare(replay.run_in_process(eng, steps), cfg, w, reqs, dtype, what)


# ------------------------------------------------------------------ the whole model, every way of cutting

@pytest.mark.parametrize("name,dtype", CASES)
def test_whole_prompts_and_first_tokens(models, name, dtype):
    reqs = requests_for(CONFIGS[name], LENGTHS[name], 1)
    check(models, name, dtype, replay.whole(reqs), reqs, "whole")


@pytest.mark.parametrize("name,dtype", CASES)
def test_prefill_against_token_by_token(models, name, dtype):
    """Every request again with its last tokens one at a time (the shortest ones entirely), 100 for the long ones:
    the windows pass over decoded tokens, and the states are carried from token to token."""
    reqs = requests_for(CONFIGS[name], LENGTHS[name], 2)
    check(models, name, dtype, replay.tail(reqs, 100), reqs, "tail")


@pytest.mark.parametrize("name,dtype", CASES)
def test_prompts_in_portions(models, name, dtype):
    """Portions of unequal sizes, then portions of two, three and five tokens and single tokens in turn: every
    portion starts inside its sequence from the state and the cache pages the portion before it left."""
    cfg = CONFIGS[name]
    reqs = requests_for(cfg, LENGTHS[name], 3)
    check(models, name, dtype, replay.pieces(reqs), reqs, "pieces")
    small = requests_for(cfg, [23, 11, 70], 4)
    plan = {}
    for i, (r, toks) in enumerate(small.items()):
        cuts, left, k = [], len(toks), i
        while left:
            c = min(left, (2, 3, 1, 2, 5)[k % 5])
            cuts.append(c); left -= c; k += 1
        plan[r] = (i, cuts)
    check(models, name, dtype, replay.scheduled(small, plan), small, "small portions")


@pytest.mark.parametrize("name,dtype", CASES)
@pytest.mark.parametrize("batch_size,fraction", [(3, 0.5), (8, 0.9)])
def test_unequal_batches_reuse_slots_and_pages(models, name, dtype, batch_size, fraction):
    """Batches one after another in a cache sized for one: slots, pages and state rows are used again, and a
    request's logits do not depend on its neighbours (compared with the plain run of each alone)."""
    reqs = requests_for(CONFIGS[name], LENGTHS[name] + LENGTHS[name][::-1], 5)
    check(models, name, dtype, replay.batched(reqs, batch_size, fraction), reqs, "batched")


@pytest.mark.parametrize("name,dtype", CASES)
def test_mixed_steps(models, name, dtype):
    """Steps that carry a fresh prompt, a later portion of another and single tokens side by side."""
    reqs = requests_for(CONFIGS[name], LENGTHS[name], 6)
    check(models, name, dtype, replay.mixed(reqs), reqs, "mixed")


@pytest.mark.parametrize("name,dtype", [("K1", "float32"), ("K1", "bfloat16"), ("K3", "bfloat16"), ("K4", "float32")])
def test_batches_of_more_rows_than_the_decode_products_fuse(models, name, dtype):
    """Twenty short requests start together and are decoded together: steps of 17 and more rows take the products and the
    residual sums that prompts take, and the recurrence walks twenty sequences side by side."""
    reqs = requests_for(CONFIGS[name], [3 + (7 * i) % 23 for i in range(20)], 13)
    check(models, name, dtype, replay.batched(reqs, 20, 0.5), reqs, "twenty rows")


@pytest.mark.parametrize("name", ["K1", "K2"])
def test_long_decoding(models, name):
    """300 tokens one by one from a one-token prompt: windows, pages given back, and states over many steps."""
    reqs = requests_for(CONFIGS[name], [301], 12)
    check(models, name, "float32", replay.tail(reqs, 300), reqs, "long decoding")


def test_a_freed_state_row_starts_from_zero(models):
    """A sequence that takes over a slot must not see the matrix states left there."""
    eng, cfg, w, _ = models[("K1", "float32")]
    reqs = requests_for(cfg, [40, 6], 8)
    steps = [{"step": 0, "entries": [{"id": "r0", "tokens": reqs["r0"], "want": [39]}], "end": ["r0"]},
             {"step": 1, "entries": [{"id": "r1", "tokens": reqs["r1"], "want": list(range(6))}], "end": ["r1"]}]
    got = replay.run_in_process(eng, steps, max_tokens=64)
    compare(got, cfg, w, reqs, "float32", "slot reuse", only_got=True)


@pytest.mark.parametrize("name", ["K1", "K3"])
@pytest.mark.parametrize("use_graph", [False, True])
def test_greedy_generation_through_the_entry_point(models, name, use_graph):
    """Engine.generate (scheduler, batches, captured decode steps) against the plain greedy loop."""
    eng, cfg, w, _ = models[(name, "float32")]
    w64 = {n: t.double() for n, t in w.items()}
    prompts = list(requests_for(cfg, [5, 1, 19, 66], 9).values())
    outs = eng.generate(prompts, max_tokens=[12, 20, 7, 9], temperature=0.0, use_graph=use_graph, stop_token_ids=[])
    for p, o, n in zip(prompts, outs, [12, 20, 7, 9]):
        assert p + o == plain.generate(p, w64, cfg, n), (len(p), o)


def test_bfloat16_generation_with_graphs_matches_eager(models):
    eng, cfg, w, _ = models[("K4", "bfloat16")]
    prompts = list(requests_for(cfg, [7, 30, 2], 11).values())
    a = eng.generate(prompts, max_tokens=10, temperature=0.0, use_graph=False, stop_token_ids=[])
    b = eng.generate(prompts, max_tokens=10, temperature=0.0, use_graph=True, stop_token_ids=[])
    assert a == b


def test_trace_replay_program(models, tmp_path):
    eng, cfg, w, folder = models[("K2", "float32")]
    reqs = requests_for(cfg, [40, 3, 77], 10)
    steps = replay.batched(reqs, 3, 0.6)
    got = replay.run_binary(folder, "float32", steps, str(tmp_path / "out"), cfg["vocab"])
    compare(got, cfg, w, reqs, "float32", "bin/trace_run")


def test_command_line_generates(models):
    import json, subprocess, sys
    eng, cfg, w, folder = models[("K3", "float32")]
    out = subprocess.run([sys.executable, "-m", "pico_engine", folder, "--prompt", "5,17,3", "--max-tokens", "6", "--temperature", "0",
                          "--dtype", "float32"], capture_output=True, text=True, cwd=replay.ROOT, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    line = [l for l in out.stdout.splitlines() if l.startswith("{")][-1]
    assert [5, 17, 3] + json.loads(line)["output"] == plain.generate([5, 17, 3], {n: t.double() for n, t in w.items()}, cfg, 6)


# ------------------------------------------------------------------ the recurrence, alone

def run_recurrence(q, k, v, dtype, lens, head_decay=None, logits=None, tau=1.0, q_scale=1.0, act="none", cuts=(1.0,), chunked=None):
    """The kernel on packed sequences of ``lens`` tokens, brought in steps that cut every sequence at the fractions
    ``cuts``; q, k [T, H, D], v [T, H, Dv] hold the sequences one after another.  Returns o [T, H, Dv] and the states."""
    from pico_engine.ops import kernels
    T, H, D = q.shape
    Dv = v.shape[2]
    B = len(lens)
    proj = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], dim=1).to(dtype).cuda().contiguous()
    z = None if logits is None else logits.reshape(T, H * D).float().cuda().contiguous()
    hd = None if head_decay is None else torch.tensor(head_decay, dtype=torch.float32).cuda()
    state = torch.full((B + 2, 5 + H * D * Dv), 3.0).cuda()               # the part's state begins at offset 5 of a slot's row
    slots = torch.tensor([b + 1 for b in range(B)], dtype=torch.int32).cuda()
    state[1:B + 1, 5:] = 0
    first = np.concatenate([[0], np.cumsum(lens)])
    out = torch.zeros(T, H * Dv)
    done = [0] * B
    for c in cuts:
        upto = [n if c == cuts[-1] else max(d, int(n * c)) for n, d in zip(lens, done)]
        rows = [b for b in range(B) if upto[b] > done[b]]
        idx = torch.cat([torch.arange(first[b] + done[b], first[b] + upto[b]) for b in rows])
        step_lens = [upto[b] - done[b] for b in rows]
        rf = torch.tensor(np.concatenate([[0], np.cumsum(step_lens)]), dtype=torch.int32).cuda()
        rl = torch.tensor(step_lens, dtype=torch.int32).cuda()
        use_chunks = (len(idx) > 2 * len(rows)) if chunked is None else chunked
        o = kernels.linear_attention(proj[idx.cuda()].contiguous(), 0, H * D, 2 * H * D, H, D, Dv, state, 5, rf, rl,
                                     slots[torch.tensor(rows).cuda()].contiguous(), use_chunks, head_decay=hd,
                                     decay_logits=None if z is None else z[idx.cuda()].contiguous(), inv_tau=1.0 / tau,
                                     q_scale=q_scale, qk_activation=act, v_activation=act)
        out[idx] = o.cpu()
        done = upto
    assert float(state[0].min()) == 3.0 and float(state[B + 1].min()) == 3.0 and float(state[:, :5].min()) == 3.0
    return out.view(T, H, Dv), state[1:B + 1, 5:].cpu().view(B, H, D, Dv)


def plain_recurrence(q, k, v, lens, decay):
    outs, states, at = [], [], 0
    for n in lens:
        o, S = plain.linear_recurrence(q[at:at + n].double(), k[at:at + n].double(), v[at:at + n].double(), decay[at:at + n].double())
        outs.append(o); states.append(S); at += n
    return torch.cat(outs), torch.stack(states)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,D,Dv", [(2, 16, 8), (3, 24, 40), (1, 64, 64), (2, 136, 12), (4, 128, 33), (1, 200, 96), (2, 128, 128), (1, 96, 72),
                                    (3, 40, 100)])
def test_recurrence_kernel_fixed_decay(dtype, H, D, Dv):
    """Sequences whose lengths fall on, before and after chunk borders, as one prompt step (chunked and token after token),
    in portions, and with the last tokens one by one; the states are compared too."""
    dt = DTYPES[dtype]
    g = torch.Generator().manual_seed(H * 1000 + D)
    lens = [1, 64, 65, 130, 2, 63, 200]
    T = sum(lens)
    q, k, v = ((torch.randn(T, H, d, generator=g) * d ** -0.25).to(dt).float() for d in (D, D, Dv))
    decay = [0.3, 1.0, 0.97, 0.999][:H] if H <= 4 else None
    dec = torch.tensor(decay).view(1, H, 1).expand(T, H, D)
    want_o, want_s = plain_recurrence(q, k, v, lens, dec)
    tol = (1e-5 if dtype == "float32" else 1e-5) * max(1.0, float(want_o.abs().max()))       # the inputs are the same rounded values
    for cuts, chunked in (((1.0,), True), ((1.0,), False), ((0.4, 0.75, 1.0), None), ((0.97, 0.98, 0.99, 1.0), None)):
        o, s = run_recurrence(q, k, v, dt, lens, head_decay=decay, cuts=cuts, chunked=chunked)
        assert (o.double() - want_o).abs().max() < tol, (cuts, chunked)
        assert (s.double() - want_s).abs().max() < tol * 10, (cuts, chunked)


@pytest.mark.parametrize("H,D,Dv,tau", [(2, 16, 8, 1.0), (3, 48, 32, 16.0), (1, 136, 24, 4.0), (2, 80, 64, 8.0), (1, 128, 160, 2.0)])
def test_recurrence_kernel_decay_per_channel(H, D, Dv, tau):
    """A learned decay per key channel and token, query scale and silu on the projections."""
    g = torch.Generator().manual_seed(D)
    lens = [70, 3, 129]
    T = sum(lens)
    q, k, v = (torch.randn(T, H, d, generator=g) for d in (D, D, Dv))
    z = 2.0 * torch.randn(T, H, D, generator=g) + 1.0
    alpha = plain.sigmoid(z.double()) ** (1.0 / tau)
    want_o, want_s = plain_recurrence(plain.silu(q.double()) * 0.25, plain.silu(k.double()), plain.silu(v.double()), lens, alpha)
    for cuts, chunked in (((1.0,), True), ((1.0,), False), ((0.5, 1.0), None)):
        o, s = run_recurrence(q, k, v, torch.float32, lens, logits=z, tau=tau, q_scale=0.25, act="silu", cuts=cuts, chunked=chunked)
        assert (o.double() - want_o).abs().max() < 2e-5 * max(1.0, float(want_o.abs().max())), (cuts, chunked)
        assert (s.double() - want_s).abs().max() < 2e-4 * max(1.0, float(want_s.abs().max()))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,D,Dv,tau", [(2, 10, 6, 1.0), (1, 37, 70, 16.0), (2, 128, 128, 16.0), (1, 256, 66, 4.0), (3, 64, 64, 0.5)])
def test_tiles_with_a_decay_per_channel(dtype, H, D, Dv, tau):
    """Chunks and runs of 16 tokens that end on, before and behind their borders, channels that fill no vector and more than one tile,
    and decays from nothing to one: the products of decays are formed forwards and lose no digits."""
    dt = DTYPES[dtype]
    g = torch.Generator().manual_seed(D)
    lens = [1, 15, 16, 17, 64, 65, 130]
    T = sum(lens)
    q, k, v = ((torch.randn(T, H, d, generator=g)).to(dt).float() for d in (D, D, Dv))
    z = 6.0 * torch.randn(T, H, D, generator=g) + 2.0
    z[::7] = -60.0
    z[3::11] = 60.0
    alpha = plain.sigmoid(z.double()) ** (1.0 / tau)
    want_o, want_s = plain_recurrence(q.double() * 0.25, k.double(), v.double(), lens, alpha)
    for cuts in ((1.0,), (0.5, 1.0)):
        o, s = run_recurrence(q, k, v, dt, lens, logits=z, tau=tau, q_scale=0.25, act="none", cuts=cuts, chunked=True)
        # float32 sums of at most 130 + 256 products whose inputs are exact in either dtype, decays good to a few 2^-24
        assert (o.double() - want_o).abs().max() < 2e-5 * max(1.0, float(want_o.abs().max())), cuts
        assert (s.double() - want_s).abs().max() < 2e-5 * max(1.0, float(want_s.abs().max())), cuts


@pytest.mark.parametrize("chunked", [False, True])
@pytest.mark.parametrize("D,pad", [(128, 0), (20, 2), (7, 0)])              # rows that do and do not allow vector reads
def test_decay_logits_of_the_rows_dtype(chunked, D, pad):
    """Logits in bfloat16 are the same numbers as those logits in float32, bit for bit, in the walk and in the tiles."""
    from pico_engine.ops import kernels
    H, Dv, lens = 3, 24, [1, 65, 17]
    T = sum(lens)
    g = torch.Generator().manual_seed(D)
    proj = torch.randn(T, 2 * H * D + H * Dv, generator=g).bfloat16().cuda()
    z = torch.empty(T * H * D + pad, dtype=torch.bfloat16, device="cuda")[pad:].view(T, H * D).copy_(4 * torch.randn(T, H * D, generator=g))
    first = torch.tensor([0, 1, 66, 83], dtype=torch.int32, device="cuda")
    rows, slots = torch.tensor(lens, dtype=torch.int32, device="cuda"), torch.arange(3, dtype=torch.int32, device="cuda")
    got = []
    for logits in (z, z.float()):
        state = torch.ones(3, H * D * Dv, device="cuda")
        got.append((kernels.linear_attention(proj, 0, H * D, 2 * H * D, H, D, Dv, state, 0, first, rows, slots, chunked,
                                             decay_logits=logits, inv_tau=0.5), state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("far", [0, 1, 63, 64, 65, 447])
def test_recurrence_keeps_a_key_from_far_back(far):
    """With decay 1 one key that matches the last query and carries a value nobody else has must come through whole
    from any distance: the first positions, chunk borders, hundreds of tokens back."""
    H, D, Dv, n = 1, 16, 8, 700
    g = torch.Generator().manual_seed(far)
    q, k, v = 0.01 * torch.randn(n, H, D, generator=g), 0.001 * torch.randn(n, H, D, generator=g), torch.randn(n, H, Dv, generator=g)
    k[far, 0] = 0; k[far, 0, 3] = 10.0
    q[-1, 0] = 0; q[-1, 0, 3] = 10.0
    v[far, 0] = 50.0                                           # the other 699 keys together add about 0.3 to the 5000
    for cuts in ((1.0,), (0.5, 0.999, 1.0)):
        o, _ = run_recurrence(q, k, v, torch.float32, [n], head_decay=[1.0], cuts=cuts)
        assert (o[-1, 0] - 5000.0).abs().max() < 2.0, (far, cuts, o[-1, 0])


# ------------------------------------------------------------------ rotation, unit norm and the cache write; the window

@pytest.mark.parametrize("pad", [5, 6])          # rows of odd and of even length (the latter let a lane take whole pairs)
@pytest.mark.parametrize("D", [24, 80, 200])
def test_rotation_norm_and_store(D, pad):
    from pico_engine.ops import kernels
    H, G, Dv, n = 3, 1, 40, 70
    g = torch.Generator().manual_seed(3)
    for dtype, tol in ((torch.float32, 2e-6), (torch.bfloat16, 1e-2)):
        for dims, norm in ((D, True), (8, True), (0, True), (16, False)):
            row = torch.randn(n, H * D + G * D + G * Dv + pad, generator=g).to(dtype)
            pos = torch.arange(100, 100 + n, dtype=torch.int32)
            freq = (50.0 ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64) / max(dims, 1)) / 3.0).float()
            kp, vp = torch.zeros(4, G, 64, D, dtype=dtype).cuda(), torch.zeros(4, G, 64, Dv, dtype=dtype).cuda()
            table = torch.tensor([[-1, 2, 0]], dtype=torch.int32).cuda()
            dev = row.cuda().contiguous()
            kernels.rotary_norm_store(dev, H, G, D, Dv, freq.cuda() if dims else None, dims, norm, 1e-5, pos.cuda(),
                                      torch.zeros(n, dtype=torch.int32).cuda(), kp, vp, table, 3)
            x = row.double()
            heads = x[:, :(H + G) * D].view(n, H + G, D)
            want = heads if not dims else plain.rotate_pairs(heads, 100, dims, 50.0, 3.0)
            # the oracle's frequencies are float64; the kernel's were rounded to float32: angles near 170 differ by 1e-5
            want = plain.rms_unit(want, 1e-5) if norm else want
            got = dev.cpu().double()
            assert (got[:, :(H + G) * D].view(n, H + G, D) - want).abs().max() < max(tol, 3e-5) * 4
            assert torch.equal(got[:, (H + G) * D:], x[:, (H + G) * D:])                      # values and the rest stay
            for t in (0, 27, 28, 69):                                                         # positions 100, 127 | 128, 169
                p = 100 + t
                page = int(table[0, p // 64])
                assert torch.equal(kp[page, :, p % 64].cpu().double().view(-1), got[t, H * D:(H + G) * D])
                assert torch.equal(vp[page, :, p % 64].cpu().double().view(-1), got[t, (H + G) * D:(H + G) * D + G * Dv])


@pytest.mark.parametrize("name,dtype", [("K1", "float32"), ("K1", "bfloat16"), ("K2", "bfloat16"), ("K2", "float32"), ("K4", "float32"), ("K4", "bfloat16")])
def test_window_edge_in_prompt_and_decoding(models, name, dtype):
    """The softmax mixer of a model alone: one key is made to dominate for the queries that follow it; it must be seen by
    the query window - 1 places after it and not by the next one, in a prompt step and token by token, with the key on
    either side of a page border."""
    from pico_engine.config.specs import GatedAttentionSpec
    eng, cfg, _, _ = models[(name, dtype)]
    layer = next(l for l in cfg["layers"] if l["type"] == "parallel")["mixer"]["left"]
    window, H, G, D, Dv = layer["mask"]["size"], layer["heads"], layer["kv_heads"], layer["dim"], layer["vdim"]
    from pico_engine.parts.attention_gated import GatedAttention
    from pico_engine.config.specs import NoPositionSpec
    part = GatedAttention(GatedAttentionSpec(hidden=8, n_heads=H, n_kv_heads=G, head_dim=D, v_head_dim=Dv, window=window, scale=1.0,
                                             position=NoPositionSpec(), prefix="", gate=None), DTYPES[dtype], "cuda")
    from pico_engine.ops import kernels
    for key_at in (5, 63, 64, 100):
        n = key_at + window + 3
        g = torch.Generator().manual_seed(key_at)
        q, k, v = 0.01 * torch.randn(n, H, D, generator=g), 0.01 * torch.randn(n, G, D, generator=g), torch.randn(n, G, Dv, generator=g)
        k[key_at] = 0; k[key_at, :, 1] = 6.0
        q[key_at + 1:] = 0; q[key_at + 1:, :, 1] = 6.0
        v[key_at] = 100.0
        dt = DTYPES[dtype]
        pages = (n + 63) // 64
        kp, vp = torch.zeros(pages + 1, G, 64, D, dtype=dt).cuda(), torch.zeros(pages + 1, G, 64, Dv, dtype=dt).cuda()
        for p in range(n):
            kp[1 + p // 64, :, p % 64] = k[p].to(dt).cuda(); vp[1 + p // 64, :, p % 64] = v[p].to(dt).cuda()
        table = torch.arange(1, pages + 1, dtype=torch.int32).view(1, -1).cuda()
        for spans in ([(0, n)], [(p, p + 1) for p in range(key_at + 1, n)]):
            for a, b in spans:
                ctx = SimpleNamespace(one_token_each=(b - a == 1), scratch={}, lens=[b - a], starts=[a], max_context=b, dtype=dt)
                pos, row = torch.arange(a, b, dtype=torch.int32).cuda(), torch.zeros(b - a, dtype=torch.int32).cuda()
                qq = q[a:b].reshape(b - a, H * D).to(dt).cuda().contiguous()
                if part.plain_kernels:
                    o = kernels.attention(qq, H * D, H, G, D, kp, vp, table, pages, pos, row, window, 1.0, ctx)
                else:
                    o = kernels.attention_headmix(qq, H * D, H, G, D, Dv, kp, vp, table, pages, pos, row, window, 1.0, None, None, ctx)
                o = o.float().cpu().view(b - a, H, Dv)
                for p in range(max(a, key_at + 1), b):
                    seen = p - key_at < window
                    assert (o[p - a].min() > 90.0) == seen and (o[p - a].max() < 10.0) == (not seen), (key_at, p, seen, o[p - a].min(), o[p - a].max())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("D", [32, 48])
def test_a_window_of_one_sees_only_the_token_itself(dtype, D):
    from pico_engine.ops import kernels
    dt = DTYPES[dtype]
    H, G, n = 4, 2, 140
    g = torch.Generator().manual_seed(D)
    q, k, v = torch.randn(n, H, D, generator=g), torch.randn(n, G, D, generator=g), torch.randn(n, G, D, generator=g).to(dt).float()
    pages = (n + 63) // 64
    kp, vp = torch.zeros(pages + 1, G, 64, D, dtype=dt).cuda(), torch.zeros(pages + 1, G, 64, D, dtype=dt).cuda()
    for p in range(n):
        kp[1 + p // 64, :, p % 64] = k[p].to(dt).cuda(); vp[1 + p // 64, :, p % 64] = v[p].to(dt).cuda()
    table = torch.arange(1, pages + 1, dtype=torch.int32).view(1, -1).cuda()
    for spans in ([(0, n)], [(p, p + 1) for p in (0, 1, 63, 64, 139)]):
        for a, b in spans:
            ctx = SimpleNamespace(one_token_each=(b - a == 1), scratch={}, lens=[b - a], starts=[a], max_context=b, dtype=dt)
            pos, row = torch.arange(a, b, dtype=torch.int32).cuda(), torch.zeros(b - a, dtype=torch.int32).cuda()
            o = kernels.attention(q[a:b].reshape(b - a, H * D).to(dt).cuda().contiguous(), H * D, H, G, D, kp, vp, table, pages, pos, row, 1, 0.3, ctx)
            want = v[a:b].repeat_interleave(H // G, dim=1)
            assert (o.float().cpu().view(b - a, H, D) - want).abs().max() < 1e-2


# ------------------------------------------------------------------ norms with gates, sums of branches, the stream

@pytest.mark.parametrize("act", ["silu", "sigmoid"])
@pytest.mark.parametrize("T,H,Dv", [(8193, 1, 4), (2731, 3, 20), (1171, 7, 64), (5462, 3, 68), (1261, 13, 128)])   # one lane a run to all of them; a last warp that is not full
def test_gated_norm_many_short_runs(T, H, Dv, act):
    """Many short runs share a warp; few have one each: the same rows through both."""
    from pico_engine.ops import kernels
    C = H * Dv
    g = torch.Generator("cpu").manual_seed(Dv)
    o, gate = torch.randn(T, C, generator=g), torch.randn(T, C + 8, generator=g).to(torch.bfloat16)
    o[5] = 0.0
    for w in (torch.randn(Dv, generator=g), torch.randn(Dv, generator=g).to(torch.bfloat16), torch.randn(Dv + 1, generator=g)[1:], None):
        w = None if w is None else torch.empty(Dv + 1, dtype=w.dtype, device="cuda")[1:].copy_(w) if w.storage_offset() else w.cuda()
        for gt in (gate.cuda(), None):
            run = lambda a, b: kernels.gated_norm(o[a:b].cuda(), Dv, w, 1e-5, None if gt is None else gt[a:b].contiguous(), 4 if gt is not None else 0, act,   # noqa: E731
                                                  torch.bfloat16)
            few = torch.cat([run(a, min(a + 4000 // H, T)) for a in range(0, T, 4000 // H)])
            # float32 sums that differ in their last places, then one rounding to bfloat16: at most a neighbour, 2^-7 of the value
            assert torch.allclose(run(0, T).float(), few.float(), rtol=2.0 ** -7, atol=1e-30)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("T,H,Dv,off", [(9, 3, 40, 7), (9, 3, 40, 8), (5, 6, 128, 0), (3, 1, 4100, 4), (4, 5, 6, 3)])
def test_gated_norm_kernel(dtype, T, H, Dv, off):
    """Norm over all heads, per head and no norm, times the gate: rows that are and are not aligned for vector accesses, runs that
    a warp, a block with registers, and a block with a loop take."""
    from pico_engine.ops import kernels
    dt = DTYPES[dtype]
    g = torch.Generator().manual_seed(1)
    o = torch.randn(T, H * Dv, generator=g) * 3
    gate = torch.randn(T, off + H * Dv, generator=g).to(dt)
    tol = 2e-6 if dtype == "float32" else 1e-2
    for group, act, fn in ((H * Dv, "sigmoid", plain.sigmoid), (Dv, "silu", plain.silu), (0, "sigmoid", plain.sigmoid)):
        w = (1 + 0.2 * torch.randn(max(group, 1), generator=g)).to(dt)
        src = o if group else o.to(dt)
        got = kernels.gated_norm(src.cuda(), group, w.cuda() if group else None, 1e-5, gate.cuda(), off, act, dt).float().cpu()
        x = src.double()
        if group:
            x = plain.norm_plain(x.view(T, -1, group), w.double(), 1e-5).reshape(T, H * Dv)
        want = x * fn(gate[:, off:].double())
        assert (got - want).abs().max() < tol * max(1.0, float(want.abs().max()))
        if group:                                           # and without a gate
            got = kernels.gated_norm(src.cuda(), group, w.cuda(), 1e-5, None, 0, "none", dt).float().cpu()
            assert (got - x).abs().max() < tol * max(1.0, float(x.abs().max()))


@pytest.mark.parametrize("T,W", [(11, 50), (5, 72), (3, 1100)])          # widths that are and are not multiples of 4, below and above 1024
def test_branch_sum_scaled_add_and_stream_vectors(T, W):
    from pico_engine.ops import kernels
    g = torch.Generator().manual_seed(2)
    x = torch.randn(T, W, generator=g)
    for dt in (torch.float32, torch.bfloat16):
        ys = [(torch.randn(T, W, generator=g) * s).to(dt) for s in (1.0, 30.0, 0.01)]
        ws = [(1 + 0.3 * torch.randn(W, generator=g)).to(dt) for _ in ys]
        for n in (1, 2, 3):
            got = kernels.normed_sum_add(x.clone().cuda(), [y.cuda() for y in ys[:n]], [w.cuda() for w in ws[:n]], 1e-5, 0.15).cpu()
            want = x.double() + 0.15 * sum(plain.norm_plain(y.double(), w.double(), 1e-5) for y, w in zip(ys[:n], ws[:n]))
            assert (got - want).abs().max() < 3e-6
        got = kernels.scaled_add(x.clone().cuda(), ys[1].cuda(), 0.3).cpu()
        assert (got - (x.double() + 0.3 * ys[1].double())).abs().max() < 1e-5
        vec = torch.randn(W, generator=g).to(dt)
        rows = torch.randn(T, W, generator=g)
        assert (kernels.add_rows(x.clone().cuda(), rows.cuda(), vec.cuda()).cpu() - (x + rows + vec.float())).abs().max() < 1e-6
        assert (kernels.add_rows(x.clone().cuda(), None, vec.cuda()).cpu() - (x + vec.float())).abs().max() < 1e-6


# ------------------------------------------------------------------ routing and the gated activation

@pytest.mark.parametrize("E,top,extra", [(8, 4, True), (5, 1, False), (3, 3, True), (70, 6, False), (1, 1, True)])
def test_expert_choice(E, top, extra):
    from pico_engine.ops import kernels
    g = torch.Generator().manual_seed(E)
    T = 37
    z = torch.randn(T, E + (1 if extra else 0), generator=g) * 3
    ids = torch.zeros(T, top, dtype=torch.int32).cuda()
    got = kernels.moe_route(z.cuda(), E, top, extra, ids).cpu()
    for t in range(T):
        order = sorted(range(E), key=lambda e: -float(z[t, e]))[:top]
        assert ids[t].tolist() == order
        p = torch.softmax(z[t, order].double(), 0)
        want = torch.zeros(E, dtype=torch.float64)
        want[order] = p
        assert (got[t, :E] - want).abs().max() < 1e-6
        assert sorted(torch.nonzero(got[t, :E]).view(-1).tolist()) == sorted(order)
        if extra:
            assert abs(float(got[t, E]) - 1 / (1 + math.exp(-float(z[t, E])))) < 1e-6


@pytest.mark.parametrize("E,top,extra,K", [(8, 4, True, 72), (3, 1, False, 50), (40, 5, True, 130)])
def test_expert_choice_from_the_stream(E, top, extra, K):
    """Norm, router product and choice in one kernel against the plain norm and router."""
    from pico_engine.ops import kernels
    g = torch.Generator().manual_seed(K)
    T = 21
    x = torch.randn(T, K, generator=g) * 3
    nw = 1 + 0.2 * torch.randn(K, generator=g)
    router = torch.randn(E + (1 if extra else 0), K, generator=g) * 3 * K ** -0.5
    ids = torch.zeros(T, top, dtype=torch.int32).cuda()
    got = kernels.moe_route_stream(x.cuda(), nw.cuda(), 1e-3, router.cuda(), E, top, extra, ids).cpu()
    z = plain.lin(router.double(), plain.norm_plain(x.double(), nw.double(), 1e-3))
    for t in range(T):
        order = sorted(range(E), key=lambda e: -float(z[t, e]))[:top]
        assert ids[t].tolist() == order
        want = torch.zeros(E, dtype=torch.float64)
        want[order] = torch.softmax(z[t, order], 0)
        assert (got[t, :E] - want).abs().max() < 1e-5
        if extra:
            assert abs(float(got[t, E]) - float(plain.sigmoid(z[t, E]))) < 1e-5


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_gated_activation_with_expert_weights(dtype):
    from pico_engine.ops import kernels
    dt = DTYPES[dtype]
    g = torch.Generator().manual_seed(4)
    T, E, ff, shared = 6, 3, 10, 7
    I = E * ff + shared
    gu = torch.randn(T, 2 * I, generator=g).to(dt)
    wts = torch.rand(T, E + 1, generator=g)
    wts[:, 1] = 0
    gu[0, ff + 2] = float("inf")                                     # a hidden unit of an expert that is not used stays out
    tol = 2e-6 if dtype == "float32" else 1e-2
    got = kernels.gated_act(gu.cuda(), "silu", wts.cuda(), ff).float().cpu()
    col = torch.tensor([min(c // ff, E) for c in range(I)])
    want = plain.silu(gu[:, :I].double()) * gu[:, I:].double() * wts.double()[:, col]
    want[:, ff:2 * ff] = 0
    assert (got - want).abs().max() < tol * 5
    got = kernels.gated_act(gu[1:].contiguous().cuda(), "gelu_tanh").float().cpu()
    want = plain.gelu_tanh(gu[1:, :I].double()) * gu[1:, I:].double()
    assert (got - want).abs().max() < tol * 5


def test_routing_of_a_model_picks_what_the_plain_router_picks(models):
    """The mixture part alone against the plain mixture, token by token."""
    eng, cfg, w, _ = models[("K1", "float32")]
    part = eng.model.layers[0].feed_forward
    g = torch.Generator().manual_seed(5)
    h = torch.randn(19, cfg["width"], generator=g)
    ctx = SimpleNamespace(dtype=torch.float32)
    got = part.apply(h.cuda(), ctx).cpu()
    want = plain.mixture(h.double(), {n: t.double() for n, t in w.items()}, "l0.mlp.", cfg["layers"][0]["mlp"])
    assert (got - want).abs().max() < 2e-5 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("odd", [float("nan"), float("inf")])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("which", ["q", "k", "v", "z"])
def test_a_token_that_is_no_number_does_not_reach_back(which, dtype, odd):
    """Chunks against the walk: what comes before the token is bit for bit what it is without it, and what comes behind is lost in the
    same places."""
    dt, H, D, Dv, lens = DTYPES[dtype], 2, 24, 70, [130, 40]
    g = torch.Generator().manual_seed(5)
    T = sum(lens)
    ins = {n: torch.randn(T, H, d, generator=g).to(dt).float() for n, d in (("q", D), ("k", D), ("v", Dv))}
    ins["z"] = torch.randn(T, H, D, generator=g) + 2
    run = lambda t, chunked: run_recurrence(t["q"], t["k"], t["v"], dt, lens, logits=t["z"], tau=16.0, chunked=chunked)
    clean = run(ins, True)[0]
    for at in (5, 63, 100):
        bad = dict(ins, **{which: ins[which].clone()})
        bad[which][at, 0, ::3] = -odd if which == "z" else odd
        (o, s), (o_walk, s_walk) = run(bad, True), run(bad, False)
        assert torch.equal(o[:at], clean[:at]) and torch.equal(o[lens[0]:], clean[lens[0]:]), at
        assert torch.equal(o.isfinite(), o_walk.isfinite()) and torch.equal(s.isfinite(), s_walk.isfinite()), at


def test_decay_logits_keep_their_digits_where_a_weight_is_stored_in_32_bits(tmp_path, monkeypatch):
    """The bfloat16 engine keeps such a weight as it is and multiplies in float32: the logits reach the recurrence as the product's float32
    sums, in prompts and in single tokens, and are the product of the rows they were made of."""
    from pico_engine.engine.engine import Engine
    from pico_engine.ops import kernels
    from pico_engine.parts import linear_attention as part
    cfg = CONFIGS["K1"]
    weights = make_weights(cfg, 40, RANKS["K1"])
    names = [n for n in weights if n.endswith(".a2")]
    for n in names:
        weights[n] = weights[n] + 2.0 ** -12 * torch.randn(weights[n].shape, generator=torch.Generator().manual_seed(1))
    eng = Engine(write_model(tmp_path / "m", cfg, weights, float32_names=names), dtype="bfloat16")
    products, logits = [], []
    linear, attend = part.linear, kernels.linear_attention
    def spy_linear(a, w, bias=None, **kw):                                             # noqa: E306
        if w.dtype == torch.float32:
            products.append(a.double() @ w.double().T + bias.double())
        return linear(a, w, bias, **kw)
    def spy_attend(*a, decay_logits=None, **kw):                                       # noqa: E306
        if decay_logits is not None:
            logits.append(decay_logits)
        return attend(*a, decay_logits=decay_logits, **kw)
    monkeypatch.setattr(part, "linear", spy_linear)
    monkeypatch.setattr(kernels, "linear_attention", spy_attend)
    replay.run_in_process(eng, replay.tail(requests_for(cfg, [70], 1), 3))
    assert len(products) == len(logits) == 4 * 3                                       # four steps, a layer that runs three times in each
    for got, want in zip(logits, products):
        # float32 sums of a rank's few products
        assert got.dtype == torch.float32 and float((got.double() - want).abs().max()) < 1e-5 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("per_channel", [False, True])
def test_chunks_in_slabs(per_channel):
    """More chunks than the scratch holds at once, sequences that end on, before and behind the borders of slabs: chunks against the walk."""
    from pico_engine.ops import kernels
    from pico_engine.ops.library import gated
    H, D, lens = 32, 128, [3000, 64, 1, 65, 4999]
    T, B = sum(lens), len(lens)
    assert gated().pe_linear_attention_slabs(T, B, H, D, D, int(per_channel)) > 1
    g = torch.Generator("cuda").manual_seed(1)
    proj = torch.randn(T, 3 * H * D, generator=g, device="cuda").bfloat16()
    decay = {"decay_logits": 2 + torch.randn(T, H * D, generator=g, device="cuda")} if per_channel else {"head_decay": torch.linspace(0.5, 0.999, H, device="cuda")}
    first, rows, slots = (torch.tensor(v, dtype=torch.int32).cuda() for v in (np.concatenate([[0], np.cumsum(lens)]), lens, range(B)))
    got = []
    for chunked in (False, True):
        state = torch.ones(B, H * D * D, device="cuda")
        got.append((kernels.linear_attention(proj, 0, H * D, 2 * H * D, H, D, D, state, 0, first, rows, slots, chunked, inv_tau=1 / 16, q_scale=D ** -0.5,
                                             **decay), state))
    for walk, chunks in zip(*got):
        # float32 sums of the same products in another order (the bound of the tests above)
        assert (walk - chunks).abs().max() < 2e-5 * max(1.0, float(walk.abs().max()))


@pytest.mark.parametrize("odd", [float("nan"), float("inf")])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("which", ["q", "k", "v"])
def test_a_token_that_is_no_number_does_not_reach_back_with_a_decay_per_head(which, dtype, odd):
    """The same with one decay a head."""
    dt, H, D, Dv, lens = DTYPES[dtype], 2, 24, 70, [130, 40]
    g = torch.Generator().manual_seed(8)
    T = sum(lens)
    ins = {n: torch.randn(T, H, d, generator=g).to(dt).float() for n, d in (("q", D), ("k", D), ("v", Dv))}
    run = lambda t, chunked: run_recurrence(t["q"], t["k"], t["v"], dt, lens, head_decay=[0.95, 0.99], chunked=chunked)
    clean = run(ins, True)[0]
    for at in (5, 63, 100):
        bad = dict(ins, **{which: ins[which].clone()})
        bad[which][at, 0, ::3] = odd
        (o, s), (o_walk, s_walk) = run(bad, True), run(bad, False)
        assert torch.equal(o[:at], clean[:at]) and torch.equal(o[lens[0]:], clean[lens[0]:]), at
        assert torch.equal(o.isfinite(), o_walk.isfinite()) and torch.equal(s.isfinite(), s_walk.isfinite()), at



def tensor_core_rows(H, D, lens, per_channel, seed, logits=torch.bfloat16):
    """Inputs of linear attention at sizes whose prompts run on the tensor cores, and a run of them."""
    from pico_engine.ops import kernels
    g = torch.Generator("cuda").manual_seed(seed)
    T, B = sum(lens), len(lens)
    proj = torch.randn(T, 3 * H * D, generator=g, device="cuda").bfloat16()
    decay = {"decay_logits": (2 + 2 * torch.randn(T, H * D, generator=g, device="cuda")).to(logits)} if per_channel else {"head_decay": torch.linspace(0.2, 0.999, H, device="cuda")}
    first, rows, slots = (torch.tensor(v, dtype=torch.int32).cuda() for v in (np.concatenate([[0], np.cumsum(lens)]), lens, range(B)))

    def run(proj, chunked, start=0.5, **more):
        state = torch.full((B, H * D * D + 3), start, device="cuda")
        o = kernels.linear_attention(proj, 0, H * D, 2 * H * D, H, D, D, state, 3, first, rows, slots, chunked, inv_tau=1 / 16, q_scale=D ** -0.5,
                                     qk_activation="none" if per_channel else "silu", **decay, **more)
        kernels.check_status(torch.device("cuda", torch.cuda.current_device()))
        return o, state[:, 3:]
    return proj, run


@pytest.mark.parametrize("per_channel,logits", [(False, None), (True, torch.bfloat16), (True, torch.float32)])
@pytest.mark.parametrize("H,D", [(1, 128), (5, 128), (2, 64), (6, 64)])
def test_linear_attention_products_on_the_tensor_cores(H, D, per_channel, logits):
    """Chunks that end on, before and behind their 64 tokens, more units than blocks: products in bfloat16 parts against the walk."""
    lens = [1, 63, 64, 65, 128, 1000, 700, 7] + [64] * (60 if H > 4 else 1)
    proj, run = tensor_core_rows(H, D, lens, per_channel, H + D, logits)
    for act in ("none", "silu"):                             # values in one part, and in three
        for walk, chunks in zip(run(proj, False, v_activation=act), run(proj, True, v_activation=act)):
            # float32 sums of the same products in another order (the bound of the tests above)
            assert (walk - chunks).abs().max() < 2e-5 * max(1.0, float(walk.abs().max())), act


@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("H,lens", [(1, [65]), (5, [200]), (7, [2048]), (3, [130, 3])])
def test_odd_heads_and_odd_chunks_on_the_tensor_cores(H, lens, per_channel):
    """An odd number of heads times an odd number of chunks: whatever lies behind their words in scratch starts on its own boundary."""
    D = 128
    proj, run = tensor_core_rows(H, D, lens, per_channel, H)
    for act in ("none", "silu"):
        for walk, chunks in zip(run(proj, False, v_activation=act), run(proj, True, v_activation=act)):
            # float32 sums of the same products in another order (the bound of the tests above)
            assert (walk - chunks).abs().max() < 2e-5 * max(1.0, float(walk.abs().max())), act


@pytest.mark.parametrize("size", [2.0 ** -122, 2.0 ** 60])
@pytest.mark.parametrize("which,what", [("v", "a head"), ("v", "some columns"), ("k", "a head"), ("q", "a token")])
@pytest.mark.parametrize("H,D,per_channel", [(2, 64, False), (2, 64, True), (3, 128, False), (3, 128, True)])
def test_numbers_of_another_size_beside_others_keep_their_digits(H, D, per_channel, which, what, size):
    """A head, some columns or a token 2^-122 or 2^60 beside numbers near one: each result to float32 of its own size."""
    lens = [130, 65]
    proj, run = tensor_core_rows(H, D, lens, per_channel, 11)
    at = "qkv".index(which) * H * D
    rows, cols = slice(None), slice(at + D, at + 2 * D)
    if what == "some columns":
        cols = slice(at + D, at + 2 * D, 3)
    if what == "a token":
        rows, cols = slice(70, 71), slice(at, at + H * D)
    proj[rows, cols] *= size
    for act in ("none", "silu") if which == "v" and size < 1 else ("none",):
        (o_walk, s_walk), (o, s) = (run(proj, chunked, 0.0, v_activation=act) for chunked in (False, True))
        o_walk, o, s_walk, s = o_walk.view(-1, H, D), o.view(-1, H, D), s_walk.view(2, H, D, D), s.view(2, H, D, D)
        # float32 sums of the same products in another order, beside the largest number of the token (of the head) and of the columns of one size
        for c in (slice(0, None, 3), slice(1, None, 3), slice(2, None, 3)):
            for walk, chunks, over in ((o_walk[..., c], o[..., c], 2), (s_walk[..., c], s[..., c], (2, 3))):
                assert ((walk - chunks).abs() <= 6e-5 * walk.abs().amax(dim=over, keepdim=True)).all(), act


def test_float32_queries_and_keys_on_the_tensor_cores():
    """Queries and keys in float32 rows of their own, which start anywhere."""
    H, D, lens = 2, 128, [200, 65]
    proj, run = tensor_core_rows(H, D, lens, False, 3)
    for pad in (0, 1):
        qk = torch.empty(sum(lens) * 2 * H * D + pad, device="cuda")[pad:].view(sum(lens), 2 * H * D)
        qk.copy_(torch.randn(sum(lens), 2 * H * D, generator=torch.Generator("cuda").manual_seed(5), device="cuda"))
        for walk, chunks in zip(run(proj, False, qk=qk), run(proj, True, qk=qk)):
            assert (walk - chunks).abs().max() < 2e-5 * max(1.0, float(walk.abs().max()))


@pytest.mark.parametrize("odd", [float("nan"), float("inf")])
@pytest.mark.parametrize("which", ["q", "k", "v"])
@pytest.mark.parametrize("H,D,per_channel", [(2, 128, False), (4, 64, False), (2, 128, True), (4, 64, True)])
def test_a_token_that_is_no_number_stays_where_it_is_on_the_tensor_cores(H, D, per_channel, which, odd):
    """Tokens in front of it and other sequences keep their bits, and the places that are lost are the walk's."""
    lens = [130, 40]
    proj, run = tensor_core_rows(H, D, lens, per_channel, 8)
    for act in ("none", "silu"):
        clean = run(proj, True, v_activation=act)[0]
        column = "qkv".index(which) * H * D
        for at in (0, 5, 63, 100):
            bad = proj.clone()
            bad[at, column: column + D: 3] = odd
            (o, s), (o_walk, s_walk) = run(bad, True, v_activation=act), run(bad, False, v_activation=act)
            assert torch.equal(o[:at], clean[:at]) and torch.equal(o[lens[0]:], clean[lens[0]:]), (at, act)
            assert torch.equal(o.isfinite(), o_walk.isfinite()) and torch.equal(s.isfinite(), s_walk.isfinite()), (at, act)


@pytest.mark.parametrize("H,D", [(3, 128), (4, 64)])
@pytest.mark.parametrize("which", ["v", "k", "z", "many"])
def test_what_a_token_that_is_no_number_does_not_reach_is_still_worked_out(H, D, which):
    """Behind such a token a unit's chunk is walked: the columns and sequences that it does not reach have their numbers, decay logits that are none
    are lost where the walk loses them, and more units than blocks of them come out right."""
    from pico_engine.ops import kernels
    lens = [130, 40] + ([64] * 150 if which == "many" else [])
    for per_channel in (True, False) if which != "z" else (True,):
        proj, run = tensor_core_rows(H, D, lens, per_channel, 9)
        if which == "z":
            T, g = sum(lens), torch.Generator("cuda").manual_seed(4)
            logits = (2 + 2 * torch.randn(T, H * D, generator=g, device="cuda")).bfloat16()
            logits[70, 5: H * D: 3] = float("nan")
            first, rows, slots = (torch.tensor(v, dtype=torch.int32).cuda() for v in (np.concatenate([[0], np.cumsum(lens)]), lens, range(len(lens))))

            def run(rows_in, chunked):
                state = torch.full((len(lens), H * D * D), 0.5, device="cuda")
                return kernels.linear_attention(rows_in, 0, H * D, 2 * H * D, H, D, D, state, 0, first, rows, slots, chunked, inv_tau=1 / 16, q_scale=D ** -0.5,
                                                decay_logits=logits), state
        elif which == "many":
            proj[5::64, 2 * H * D: 3 * H * D: 7] = float("nan")
        else:
            column = "qkv".index(which) * H * D
            proj[70, column + 3: column + D: 5] = float("inf") if which == "k" else float("nan")
        for walk, chunks in zip(run(proj, False), run(proj, True)):
            there = walk.isfinite()
            assert torch.equal(there, chunks.isfinite()) and there.any() and not there.all()
            # float32 sums of the same products in another order (the bound of the tests above)
            assert (walk - chunks)[there].abs().max() < 2e-5 * max(1.0, float(walk[there].abs().max()))


@pytest.mark.parametrize("per_channel", [False, True])
def test_a_sequence_that_is_no_number_does_not_hold_up_the_others(per_channel):
    """A batch's step with one such sequence takes about as long as without it: 1.1 to 2 times where a walk from memory took 20 to 80."""
    lens = [1024] * 4
    proj, run = tensor_core_rows(16, 128, lens, per_channel, 2)
    bad = proj.clone()
    bad[5] = float("nan")

    def time(rows):
        run(rows, True)
        best = float("inf")
        for _ in range(5):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            run(rows, True)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best
    assert time(bad) < 4 * time(proj)


@pytest.mark.parametrize("per_channel", [False, True])
def test_odd_heads_in_slabs_on_the_tensor_cores(per_channel):
    """More chunks than the scratch holds at once, an odd number of them a slab and of heads; sequences that begin in one slab and end in the next."""
    from pico_engine.ops.library import gated
    H, D, lens = 5, 128, [5000, 64, 1, 5000, 4780]
    kind = int(per_channel) | 2
    chunks = -(-sum(lens) // 64) + len(lens)
    assert gated().pe_linear_attention_slabs(sum(lens), len(lens), H, D, D, kind | 4) == 2 and -(-chunks // 2) % 2
    proj, run = tensor_core_rows(H, D, lens, per_channel, 6)
    for walk, out in zip(run(proj, False, v_activation="silu"), run(proj, True, v_activation="silu")):
        # float32 sums of the same products in another order (the bound of the tests above)
        assert (walk - out).abs().max() < 2e-5 * max(1.0, float(walk.abs().max()))


@pytest.mark.parametrize("H,D,per_channel,most_o,most_state", [(14, 64, False, 1.6e-7, 1.06e-7), (14, 64, True, 1.7e-7, 1.35e-7), (3, 128, False, 2.0e-7, 1.0e-7), (3, 128, True, 2.0e-7, 1.4e-7)])
def test_errors_are_no_larger_than_multiply_adds(H, D, per_channel, most_o, most_state):
    """Outputs and states against 64 bits, beside their norms, means over four inputs; the bounds are what the multiply-add tiles leave of such inputs."""
    from pico_engine.ops import kernels
    T, errors = 200, []
    first, rows, slots = (torch.tensor(v, dtype=torch.int32).cuda() for v in ([0, T], [T], [0]))
    for seed in range(4):
        g = torch.Generator("cuda").manual_seed(seed)
        proj, z = torch.randn(T, 3 * H * D, generator=g, device="cuda").bfloat16(), (1.5 * torch.randn(T, H * D, generator=g, device="cuda")).bfloat16()
        fixed, state = torch.tensor([1 - 2.0 ** -(3 + h % 6) for h in range(H)], device="cuda"), torch.zeros(1, H * D * D, device="cuda")
        how = dict(decay_logits=z, inv_tau=1 / 16, q_scale=D ** -0.5) if per_channel else dict(head_decay=fixed, qk_activation="silu", v_activation="silu")
        o = kernels.linear_attention(proj, 0, H * D, 2 * H * D, H, D, D, state, 0, first, rows, slots, True, **how)
        q, k, v = (t.double().view(T, H, D) for t in proj.split(H * D, 1))
        if per_channel:
            q, decay = q * D ** -0.5, (torch.sigmoid(z.double()) ** (1 / 16)).view(T, H, D)
        else:
            q, k, v = (torch.nn.functional.silu(t) for t in (q, k, v))
            decay = fixed.double().view(1, H, 1).expand(T, H, D)
        S, want = torch.zeros(H, D, D, dtype=torch.float64, device="cuda"), torch.empty_like(v)
        for t in range(T):
            S = decay[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None]
            want[t] = (q[t][:, None] @ S)[:, 0]
        errors.append([float((o.view(T, H, D) - want).norm() / want.norm()), float((state.view(H, D, D) - S).norm() / S.norm())])
    e_o, e_state = np.mean(errors, 0)
    assert e_o < most_o and e_state < most_state, (e_o, e_state)
