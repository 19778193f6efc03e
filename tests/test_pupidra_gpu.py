"""Pupidra on the GPU against the plain implementation: each mechanism's kernel alone on inputs that show a fault, and the
whole model through the library's step function, cache, scheduler and entry points, in both dtypes, for every way of
cutting requests into steps."""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import pytest
import torch

import plain_pupidra as plain
import replay
from conftest import write_model
from pupidra_models import CONFIGS, make_weights, plain_logits, requests_for

pytestmark = pytest.mark.gpu

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}
CASES = [(n, d) for n in sorted(CONFIGS) for d in ("float32", "bfloat16")]
LENGTHS = {"P1": [1, 2, 3, 47, 70, 131, 64, 5], "P2": [65, 1, 150, 9, 33, 2], "P3": [3, 129, 31, 64, 1, 70], "P4": [4, 1, 290, 17, 66, 135]}


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    """{(config, dtype): (engine, cfg, weights, folder)}."""
    from pico_engine.engine.engine import Engine
    root = tmp_path_factory.mktemp("pupidra")
    out = {}
    for k, (name, cfg) in enumerate(sorted(CONFIGS.items())):
        weights = make_weights(cfg, 60 + k)
        folder = write_model(root / name, cfg, weights)
        for dtype in DTYPES:
            out[(name, dtype)] = (Engine(folder, dtype=dtype), cfg, weights, folder)
    return out


def compare(got, cfg, w, reqs, dtype, what, only_got=False):
    """Against the plain logits.  float32: every place, by the rule of the engine tests.  bfloat16: without the places where
    the plain router's choice was a close call and the two places behind each (which weigh that place's keys, values and
    convolution inputs most, and inherit another choice of experts there); of the others none may be off by more than a tenth of the logits' size, and
    at most one in a hundred by more than the engine tests' 4e-2 (a sublayer's output is normed before it is added, so a
    small output carries its rounding at full size into the stream: a few places lie just above the rule of the pre-norm designs)."""
    close = set()
    want = plain_logits(cfg, w, reqs, close)
    if only_got:
        want = {k: v for k, v in want.items() if k in got}
    if dtype != "bfloat16":
        return replay.compare(got, want, dtype, what)
    assert set(got) == set(want), (what, sorted(set(want) - set(got))[:5], sorted(set(got) - set(want))[:5])
    close |= {(r, p + d) for r, p in close for d in (1, 2)}
    assert len(close & set(want)) < 0.6 * len(want)
    over = []
    for key in sorted(set(want) - close, key=lambda k: (str(k[0]), k[1])):
        scale = max(1.0, float(np.abs(want[key]).max()))
        err = float(np.abs(np.asarray(got[key], dtype=np.float64) - want[key]).max()) / scale
        assert err <= 1e-1, f"{what}: request {key[0]!r} position {key[1]}: max error {err:.3e} of the logits' size {scale:.3f}"
        if err > 4e-2:
            over.append((key, round(err, 4)))
    assert len(over) <= max(1, len(set(want) - close) // 100), (what, over[:8])


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
    """Every request again with its last tokens one at a time (the shortest ones entirely), 100 for the long ones: the
    windows pass over decoded tokens, pages behind them are given back while kept ones stay, and the states and the
    token before are carried from step to step."""
    reqs = requests_for(CONFIGS[name], LENGTHS[name], 2)
    check(models, name, dtype, replay.tail(reqs, 100), reqs, "tail")


@pytest.mark.parametrize("name,dtype", CASES)
def test_prompts_in_portions(models, name, dtype):
    """Portions of unequal sizes, then portions of two, three and five tokens and single tokens in turn: every portion starts
    inside its sequence from the state and the cache pages the portion before it left."""
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
    """Batches one after another in a cache sized for one: slots, pages and state rows are used again, and a request's logits
    do not depend on its neighbours (compared with the plain run of each alone)."""
    reqs = requests_for(CONFIGS[name], LENGTHS[name] + LENGTHS[name][::-1], 5)
    check(models, name, dtype, replay.batched(reqs, batch_size, fraction), reqs, "batched")


@pytest.mark.parametrize("name,dtype", CASES)
def test_mixed_steps(models, name, dtype):
    """Steps that carry a fresh prompt, a later portion of another and single tokens side by side."""
    reqs = requests_for(CONFIGS[name], LENGTHS[name], 6)
    check(models, name, dtype, replay.mixed(reqs), reqs, "mixed")


@pytest.mark.parametrize("name,dtype", [("P1", "float32"), ("P1", "bfloat16"), ("P4", "bfloat16"), ("P3", "float32")])
def test_batches_of_more_rows_than_the_decode_products_fuse(models, name, dtype):
    """Twenty short requests start together and are decoded together: steps of 17 and more rows take the products that prompts
    take, and the recurrence walks twenty sequences side by side."""
    reqs = requests_for(CONFIGS[name], [3 + (7 * i) % 23 for i in range(20)], 13)
    check(models, name, dtype, replay.batched(reqs, 20, 0.5), reqs, "twenty rows")


@pytest.mark.parametrize("name", ["P1", "P3", "P4"])
def test_long_decoding(models, name):
    """300 tokens one by one from a one-token prompt: windows, kept first tokens, pages given back, and states over many steps."""
    reqs = requests_for(CONFIGS[name], [301], 12)
    check(models, name, "float32", replay.tail(reqs, 300), reqs, "long decoding")


def test_a_freed_slot_starts_from_nothing(models):
    """A sequence that takes over a slot must not see the matrix states, the convolution's inputs or the last token left there."""
    eng, cfg, w, _ = models[("P1", "float32")]
    reqs = requests_for(cfg, [40, 6], 8)
    steps = [{"step": 0, "entries": [{"id": "r0", "tokens": reqs["r0"], "want": [39]}], "end": ["r0"]},
             {"step": 1, "entries": [{"id": "r1", "tokens": reqs["r1"], "want": list(range(6))}], "end": ["r1"]}]
    got = replay.run_in_process(eng, steps, max_tokens=64)
    compare(got, cfg, w, reqs, "float32", "slot reuse", only_got=True)


@pytest.mark.parametrize("name", ["P1", "P4"])
@pytest.mark.parametrize("use_graph", [False, True])
def test_greedy_generation_through_the_entry_point(models, name, use_graph):
    """Engine.generate (scheduler, batches, captured decode steps) against the plain greedy loop."""
    eng, cfg, w, _ = models[(name, "float32")]
    w64 = {n: t.double() for n, t in w.items()}
    prompts = list(requests_for(cfg, [5, 1, 19, 66], 9).values())
    news = [12, 20, 7, 9]
    outs = eng.generate(prompts, max_tokens=news, temperature=0.0, use_graph=use_graph, stop_token_ids=[])
    for p, o, n in zip(prompts, outs, news):
        with torch.no_grad():
            assert o == plain.greedy(p, cfg, w64, n), (len(p), o)


def test_bfloat16_generation_with_graphs_matches_eager(models):
    eng, cfg, w, _ = models[("P3", "bfloat16")]
    prompts = list(requests_for(cfg, [7, 30, 2], 11).values())
    a = eng.generate(prompts, max_tokens=10, temperature=0.0, use_graph=False, stop_token_ids=[])
    b = eng.generate(prompts, max_tokens=10, temperature=0.0, use_graph=True, stop_token_ids=[])
    assert a == b


def test_trace_replay_program(models, tmp_path):
    eng, cfg, w, folder = models[("P2", "float32")]
    reqs = requests_for(cfg, [40, 3, 77], 10)
    steps = replay.batched(reqs, 3, 0.6)
    got = replay.run_binary(folder, "float32", steps, str(tmp_path / "out"), cfg["vocab"])
    compare(got, cfg, w, reqs, "float32", "bin/trace_run")


def test_command_line_generates(models):
    import json, subprocess, sys
    eng, cfg, w, folder = models[("P1", "float32")]
    out = subprocess.run([sys.executable, "-m", "pico_engine", folder, "--prompt", "5,17,3", "--max-tokens", "6", "--temperature", "0",
                          "--dtype", "float32"], capture_output=True, text=True, cwd=replay.ROOT, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    line = [l for l in out.stdout.splitlines() if l.startswith("{")][-1]
    with torch.no_grad():
        assert json.loads(line)["output"] == plain.greedy([5, 17, 3], cfg, {n: t.double() for n, t in w.items()}, 6)


# ------------------------------------------------------------------ attention with a distance bias, a window and kept first keys, alone

def paged(k, dt, first_page=1):
    """k [n, G, D] as cache pages [pages + first_page, G, 64, D] and the page table of one sequence."""
    n, G, D = k.shape
    pages = (n + 63) // 64
    pool = torch.zeros(pages + first_page, G, 64, D, dtype=dt).cuda()
    for p in range(n):
        pool[first_page + p // 64, :, p % 64] = k[p].to(dt).cuda()
    return pool, torch.arange(first_page, pages + first_page, dtype=torch.int32).view(1, -1).cuda()


def run_attention(q, kp, vp, table, dt, spans, window, keep, scale, slopes, Dv, values_in_keys=False):
    """``kernels.attention_headmix`` for the query positions of ``spans`` (each a step of one sequence); q [n, H, D]."""
    from pico_engine.ops import kernels
    n, H, D = q.shape
    G = kp.shape[1]
    out = torch.zeros(n, H * Dv)
    sl = None if slopes is None else torch.tensor(slopes, dtype=torch.float32).cuda()
    for a, b in spans:
        ctx = SimpleNamespace(one_token_each=(b - a == 1), scratch={}, lens=[b - a], starts=[a], max_context=b, dtype=dt)
        pos, row = torch.arange(a, b, dtype=torch.int32).cuda(), torch.zeros(b - a, dtype=torch.int32).cuda()
        qq = q[a:b].reshape(b - a, H * D).to(dt).cuda().contiguous()
        o = kernels.attention_headmix(qq, H * D, H, G, D, Dv, kp, vp, table, table.shape[1], pos, row, window, scale, None, None, ctx,
                                      slopes=sl, keep_first=keep, values_in_keys=values_in_keys)
        out[a:b] = o.float().cpu()
    return out.view(n, H, Dv)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,G,D,Dv,window,keep", [(6, 2, 32, 16, 40, 5), (3, 1, 24, 12, 2, 1), (8, 1, 64, 64, 130, 70), (2, 2, 16, 16, 64, 64),
                                                  (4, 4, 16, 24, None, 0), (4, 2, 48, 40, 70, 0), (2, 1, 128, 128, 65, 3)])
def test_biased_attention_kernel(dtype, H, G, D, Dv, window, keep):
    """Random queries, keys and values against the plain function: as one prompt, in portions, and the last 80 tokens one by one."""
    dt = DTYPES[dtype]
    n = 230
    g = torch.Generator().manual_seed(H * 100 + D)
    q, k, v = ((torch.randn(n, h, d, generator=g)).to(dt).float() for h, d in ((H, D), (G, D), (G, Dv)))
    scale = 0.5 * D ** -0.5
    want = plain.biased_attention(q.double(), k.double(), v.double(), scale, window, keep)
    kp, table = paged(k, dt)
    vp, _ = paged(v, dt)
    tol = 2e-5 if dtype == "float32" else 2e-2
    for spans in ([(0, n)], [(0, 3), (3, 70), (70, 72), (72, 200), (200, n)], [(0, 150)] + [(p, p + 1) for p in range(150, n)]):
        got = run_attention(q, kp, vp, table, dt, spans, window, keep, scale, plain.distance_slopes(H), Dv)
        assert (got.double() - want).abs().max() < tol * max(1.0, float(want.abs().max())), spans[:2]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,G,D,Dv,window,keep", [(6, 2, 32, 16, 40, 5), (3, 1, 24, 12, 2, 1), (8, 1, 64, 64, 130, 70), (2, 2, 16, 16, 64, 64),
                                                  (2, 1, 64, 64, 66, 3), (2, 2, 128, 128, 40, 65)])
def test_window_and_kept_edges_in_prompt_and_decoding(dtype, H, G, D, Dv, window, keep):
    """One key is made to dominate for the queries that follow it.  A key behind the kept ones must be seen by the query
    window - 1 places after it and not by the next one; the last kept key must be seen from everywhere and the first key
    that is not kept only inside its window; in a prompt step and token by token, with the key on either side of a page border."""
    dt = DTYPES[dtype]
    for key_at in sorted({keep - 1, keep, keep + 58, keep + 59, 63 + keep, 64 + keep, 127 + keep} - {-1}):
        n = key_at + window + 70
        g = torch.Generator().manual_seed(key_at)
        q, k, v = 0.01 * torch.randn(n, H, D, generator=g), 0.01 * torch.randn(n, G, D, generator=g), torch.randn(n, G, Dv, generator=g)
        k[key_at] = 0; k[key_at, :, 1] = 30.0
        q[key_at + 1:] = 0; q[key_at + 1:, :, 1] = 30.0              # a score of 900 against a distance bias of 0.5 a place at most
        v[key_at] = 100.0
        kp, table = paged(k, dt)
        vp, _ = paged(v, dt)
        for spans in ([(0, n)], [(0, key_at + 1)] + [(p, p + 1) for p in range(key_at + 1, n)]):
            got = run_attention(q, kp, vp, table, dt, spans, window, keep, 1.0, plain.distance_slopes(H), Dv)
            for p in range(key_at + 1, n):
                seen = p - key_at < window or key_at < keep
                assert ((got[p] - 100.0).abs().max() < 1.0) == seen, (key_at, p, len(spans), got[p].abs().max())


@pytest.mark.parametrize("H,G,D,window,keep", [(4, 2, 64, 100, 70), (2, 1, 128, 65, 3), (2, 2, 64, 64, 0), (3, 1, 64, None, 0),
                                               (2, 2, 128, 200, 128), (2, 1, 64, 300, 1)])
def test_long_prompts_in_bfloat16_at_head_sizes_of_the_tensor_memory_kernel(H, G, D, window, keep):
    """Prompts long enough that the pages of the kept first keys and the pages of the window lie apart, whole, in portions
    that begin and end off the borders of pages and of the kernel's runs of tokens, and with the last 330 tokens one by one."""
    dt, n = torch.bfloat16, 900
    g = torch.Generator().manual_seed(H * 100 + D + (window or 0))
    q, k, v = ((torch.randn(n, h, D, generator=g)).to(dt).float() for h in (H, G, G))
    scale = 0.7 * D ** -0.5
    want = plain.biased_attention(q.double(), k.double(), v.double(), scale, window, keep)
    kp, table = paged(k, dt)
    vp, _ = paged(v, dt)
    for spans in ([(0, n)], [(0, 130), (130, 133), (133, 517), (517, n)], [(0, 570)] + [(p, p + 1) for p in range(570, n)]):
        got = run_attention(q, kp, vp, table, dt, spans, window, keep, scale, plain.distance_slopes(H), D)
        assert (got.double() - want).abs().max() < 2e-2 * max(1.0, float(want.abs().max())), spans[:2]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("far", [0, 1, 63, 64, 65, 447])
def test_a_key_from_far_back(dtype, far):
    """Without a window, and in the kernel's form for latent rows (one key head whose first entries are the value), one key
    that matches the last query must come through from any distance, although the distance bias counts against it."""
    dt = DTYPES[dtype]
    H, n = 4, 700
    for G, D, Dv, in_keys in ((2, 32, 24, False), (1, 48, 40, True)):
        g = torch.Generator().manual_seed(far)
        q, k, v = 0.01 * torch.randn(n, H, D, generator=g), 0.01 * torch.randn(n, G, D, generator=g), torch.randn(n, G, Dv, generator=g)
        k[far] = 0; k[far, :, D - 1] = 40.0
        q[-1] = 0; q[-1, :, D - 1] = 40.0                            # 1600 against at most 0.5 * 700
        if in_keys:
            v = k[:, :, :Dv].clone()
            v[far] = k[far, :, :Dv] = 8.0
            k[far, :, D - 1] = 40.0
        else:
            v[far] = 8.0
        kp, table = paged(k, dt)
        vp = None if in_keys else paged(v, dt)[0]
        for spans in ([(0, n)], [(n - 1, n)]):
            got = run_attention(q, kp, vp, table, dt, spans, None, 0, 1.0, None if in_keys else plain.distance_slopes(H), Dv, in_keys)
            assert (got[-1] - 8.0).abs().max() < 0.1, (far, in_keys, got[-1])


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("H,width,rank,window", [(1, 64, 64, None), (3, 96, 64, 70), (14, 160, 128, None), (5, 192, 128, 128), (2, 256, 192, None),
                                                 (16, 256, 192, 200), (2, 208, 192, 1)])
def test_prompts_over_low_rank_rows(H, width, rank, window, gated):
    """The tcgen05 kernel at every number of panels: whole prompts and portions that begin and end off the borders of pages and of runs
    of 128 tokens, several sequences in a step, pages that the window has left given back, a gate a head."""
    from pico_engine.ops import kernels
    g = torch.Generator().manual_seed(H * 1000 + width)
    lens, dt = [1, 63, 129, 470], torch.bfloat16
    scale = 1.5 * width ** -0.5
    q, k = (torch.randn(sum(lens), h, width, generator=g).to(dt).float() for h in (H, 1))
    logits = (2 * torch.randn(sum(lens), H + 3, generator=g)).to(dt)
    pages = sum((n + 63) // 64 for n in lens)
    pool = torch.full((pages + 1, 1, 64, width), 3.0, dtype=dt)          # what no sequence has written is not seen
    table = torch.full((len(lens), 9), -1, dtype=torch.int32)
    want, at, page = [], 0, 1
    for b, n in enumerate(lens):
        for j in range((n + 63) // 64):
            m = min(64, n - 64 * j)
            pool[page, 0, :m], table[b, j], page = k[at + 64 * j: at + 64 * j + m, 0].to(dt), page, page + 1
        i, j = torch.arange(n)[:, None], torch.arange(n)[None]
        seen = (j <= i) if window is None else (j <= i) & (i - j < window)
        s = torch.einsum("ihd,jd->hij", q[at: at + n].double(), k[at: at + n, 0].double()) * scale
        w = torch.softmax(s.masked_fill(~seen, float("-inf")), -1)
        want.append(torch.einsum("hij,jd->ihd", w, k[at: at + n, 0, :rank].double()))
        at += n
    want = torch.cat(want)
    if gated:
        want = want * torch.sigmoid(logits[:, 2: 2 + H].double())[..., None]
    want = want.reshape(-1, H * rank)
    first = np.concatenate([[0], np.cumsum(lens)])
    for cuts in ([(0, n) for n in lens], [(n // 3, n) for n in lens], [(n - min(n, 2), n) for n in lens]):
        idx = torch.cat([torch.arange(first[b] + lo, first[b] + hi) for b, (lo, hi) in enumerate(cuts)])
        tab = table.clone()
        if window is not None:
            for b, (lo, _) in enumerate(cuts):
                tab[b, : max(0, lo - window + 1) // 64] = -1
        ctx = SimpleNamespace(one_token_each=False, scratch={}, lens=[hi - lo for lo, hi in cuts], starts=[lo for lo, _ in cuts], dtype=dt)
        got = kernels.attention_latent_prompt(q[idx].reshape(len(idx), -1).to(dt).cuda(), H * width, H, width, rank, pool.cuda(), tab.cuda(), tab.shape[1],
                                              window, scale, ctx, logits[idx].cuda() if gated else None, 2)
        kernels.check_status(torch.device("cuda", torch.cuda.current_device()))
        # weights and results are rounded to bfloat16 (2^-9 each), values reach four: 2e-2 as for the other bfloat16 attention kernels
        assert (got.double().cpu() - want[idx]).abs().max() < 2e-2 * max(1.0, float(want.abs().max())), cuts


# ------------------------------------------------------------------ the state-space mixer's kernels, alone

def run_state_space(proj, m, conv_w, conv_b, dt_bias, a_log, d_skip, norm_w, eps, dt, lens, cuts, chunked=False):
    """Convolution, recurrence and gated norm on packed sequences of ``lens`` tokens (rows of proj = z | x | B | C | dt), brought
    in steps that cut every sequence at the fractions ``cuts``; returns [T, inner] and the final matrix states."""
    from pico_engine.ops import kernels
    H, P, N, G, taps, groups = m["heads"], m["vdim"], m["state"], m["groups"], m["conv"], m["norm_groups"]
    inner, conv = H * P, H * P + 2 * G * N
    T, B = proj.shape[0], len(lens)
    elems = kernels.state_space_elems(H, P, N)
    state = torch.full((B + 2, 5 + elems + (taps - 1) * conv), 3.0).cuda()      # the part's state begins at offset 5 of a slot's row
    state[1:B + 1, 5:] = 0
    slots = torch.tensor([b + 1 for b in range(B)], dtype=torch.int32).cuda()
    dev = proj.to(dt).cuda().contiguous()
    cw, cb, nw = conv_w.to(dt).cuda(), conv_b.to(dt).cuda(), norm_w.to(dt).cuda()
    f32 = [t.float().cuda() for t in (dt_bias, a_log, d_skip)]
    first = np.concatenate([[0], np.cumsum(lens)])
    out = torch.zeros(T, inner)
    done = [0] * B
    for c in cuts:
        upto = [n if c == cuts[-1] else max(d, int(n * c)) for n, d in zip(lens, done)]
        rows = [b for b in range(B) if upto[b] > done[b]]
        idx = torch.cat([torch.arange(first[b] + done[b], first[b] + upto[b]) for b in rows])
        step_lens = [upto[b] - done[b] for b in rows]
        rf = torch.tensor(np.concatenate([[0], np.cumsum(step_lens)]), dtype=torch.int32).cuda()
        rl = torch.tensor(step_lens, dtype=torch.int32).cuda()
        tr = torch.tensor(np.repeat(np.arange(len(rows)), step_lens), dtype=torch.int32).cuda()
        sl = slots[torch.tensor(rows).cuda()].contiguous()
        p = dev[idx.cuda()].contiguous()
        xbc = kernels.conv_silu(p, inner, conv, cw, cb, state, 5 + elems, tr, rf, rl, sl)
        y = kernels.state_space_scan(xbc, p, inner + conv, *f32, state, 5, rf, rl, sl, H, P, N, G, chunked=chunked)
        out[idx] = kernels.gate_norm(y, inner // groups, p, 0, nw, eps).float().cpu()
        done = upto
    assert float(state[0].min()) == 3.0 and float(state[B + 1].min()) == 3.0 and float(state[:, :5].min()) == 3.0
    return out


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("shift", [0, 1])
def test_convolution_of_runs_where_rows_meet(dtype, taps, shift):
    """Rows that begin and end at every place of a run of eight tokens, one to nine tokens long and longer, from a state that is not zero, with
    weights off the boundary that four of them are read from: against float64.  A sum has taps + 1 roundings of at most the sum of its
    terms' magnitudes (2^-24 each), which silu passes on at most 1.1-fold and rounds to a few 2^-24 of itself."""
    from pico_engine.ops import kernels
    dt, C, ld, off = DTYPES[dtype], 1280, 1288, 4
    lens = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 3, 1, 1, 13, 300, 64, 27]
    T, B = sum(lens), len(lens)
    assert T * C >= 500000 and T >= 8 * B                        # the sizes that runs take
    g = torch.Generator().manual_seed(taps)
    proj = torch.randn(T, ld, generator=g).to(dt)
    w, bias = (torch.randn(*n, generator=g).to(dt).cuda().view(-1)[shift:] for n in ((C * taps + shift,), (C + shift,)))
    state = torch.randn(B + 1, (taps - 1) * C, generator=g).cuda()
    slots = torch.arange(B, 0, -1, dtype=torch.int32).cuda()
    first = np.concatenate([[0], np.cumsum(lens)])
    old = state.double().cpu()
    got = kernels.conv_silu(proj.cuda(), off, C, w.view(C, taps), bias, state, 0, torch.tensor(np.repeat(np.arange(B), lens), dtype=torch.int32).cuda(),
                            torch.tensor(first, dtype=torch.int32).cuda(), torch.tensor(lens, dtype=torch.int32).cuda(), slots).double().cpu()
    w64, b64 = w.view(C, taps).double().cpu(), bias.double().cpu()
    for b, n in enumerate(lens):
        rows = proj[first[b]: first[b] + n, off: off + C].double()
        u = torch.cat([old[B - b].view(taps - 1, C).flip(0), rows])          # entry k of a state: the input k + 1 places before the step
        terms = torch.stack([w64[:, j] * u[j: j + n] for j in range(taps)])
        v = terms.sum(0) + b64
        err = (got[first[b]: first[b] + n] - v * torch.sigmoid(v)).abs()
        assert (err <= 2.0 ** -24 * (1.1 * (taps + 1) * (terms.abs().sum(0) + b64.abs()) + 8 * v.abs())).all(), (b, n)
        assert torch.equal(state[B - b].double().cpu().view(taps - 1, C), u.flip(0)[: taps - 1])


def test_convolution_of_weights_just_written():
    """Weights that the kernel in front writes: none is read before it is there."""
    from pico_engine.ops import kernels
    T, C, taps = 1000, 1024, 4
    g = torch.Generator().manual_seed(1)
    rnd = lambda *n: torch.randn(*n, generator=g)
    proj, state, ids = rnd(T, C).cuda(), torch.zeros(1, (taps - 1) * C, device="cuda"), torch.arange(C, dtype=torch.int32).flip(0).cuda()
    bias, zeros, one = rnd(C).cuda(), torch.zeros(T, dtype=torch.int32, device="cuda"), torch.tensor([0, T], dtype=torch.int32, device="cuda")
    run = lambda w: kernels.conv_silu(proj, 0, C, w, bias, torch.zeros_like(state), 0, zeros, one, one[1:], zeros[:1])
    tables = [rnd(C, taps).cuda() for _ in range(8)]
    want = [run(t.flip(0)) for t in tables]
    w = torch.zeros(C, taps, device="cuda")
    states = [state.clone() for _ in tables]
    torch.cuda.synchronize()
    got = [kernels.conv_silu(proj, 0, C, kernels.embed(t, ids, out=w), bias, s, 0, zeros, one, one[1:], zeros[:1]) for t, s in zip(tables, states)]
    assert all(torch.equal(g, v) for g, v in zip(got, want))


def plain_state_space(proj, m, conv_w, conv_b, dt_bias, a_log, d_skip, norm_w, eps, lens):
    H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * P
    outs, at = [], 0
    for n in lens:
        pr = proj[at:at + n].double()
        z, xbc, dtr = pr[:, :inner], pr[:, inner: 2 * inner + 2 * G * N], pr[:, 2 * inner + 2 * G * N:]
        xbc = plain.silu(plain.causal_conv(xbc, conv_w.double(), conv_b.double()))
        y = plain.ssm_recurrence(xbc[:, :inner].reshape(n, H, P), xbc[:, inner: inner + G * N].reshape(n, G, N),
                                 xbc[:, inner + G * N:].reshape(n, G, N), plain.softplus(dtr + dt_bias.double()),
                                 -torch.exp(a_log.double()), d_skip.double()).reshape(n, inner) * plain.silu(z)
        groups = m["norm_groups"]
        outs.append(plain.rms_unit(y.view(n, groups, inner // groups), eps).reshape(n, inner) * norm_w.double())
        at += n
    return torch.cat(outs)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,P,N,G,taps,groups", [(4, 16, 24, 2, 3, 4), (2, 8, 40, 1, 2, 1), (3, 5, 7, 3, 1, 3), (4, 32, 128, 4, 4, 2),
                                                  (2, 64, 16, 2, 4, 1), (1, 40, 200, 1, 5, 8), (6, 24, 64, 3, 4, 2)])
def test_state_space_kernels(dtype, H, P, N, G, taps, groups):
    """Sequences of many lengths as one prompt step, in portions, and with the last tokens one by one; a sequence's walk and the
    three passes over chunks of 64."""
    dt = DTYPES[dtype]
    m = {"heads": H, "vdim": P, "state": N, "groups": G, "conv": taps, "norm_groups": groups}
    g = torch.Generator().manual_seed(H * 1000 + N)
    lens = [1, 2, 9, 70, 3, 131, 64, 200]
    T, inner, conv = sum(lens), H * P, H * P + 2 * G * N
    r = lambda *s: torch.randn(*s, generator=g)
    rounded = lambda t: t.to(dt).float()
    proj = rounded(r(T, 2 * inner + 2 * G * N + H))
    conv_w, conv_b, norm_w = rounded(0.6 * r(conv, taps)), rounded(0.3 * r(conv)), rounded(1 + 0.1 * r(inner))
    dt_bias, a_log, d_skip = r(H) - 1.0, 0.7 * r(H) - 0.5, 1 + 0.3 * r(H)
    args = (m, conv_w, conv_b, dt_bias, a_log, d_skip, norm_w, 1e-5)
    want = plain_state_space(proj, *args, lens)
    tol = (3e-5 if dtype == "float32" else 1.5e-2) * max(1.0, float(want.abs().max()))
    for cuts in ((1.0,), (0.4, 0.75, 1.0), (0.97, 0.98, 0.99, 1.0)):
        for chunked in (False, True):
            got = run_state_space(proj, *args, dt, lens, cuts, chunked)
            assert (got.double() - want).abs().max() < tol, (cuts, chunked)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,P,N,G,taps,groups", [(2, 72, 130, 1, 4, 1), (4, 64, 128, 2, 3, 2), (1, 68, 33, 1, 2, 1), (20, 64, 20, 1, 4, 1), (36, 64, 4, 2, 4, 1)])
def test_state_space_kernels_at_the_edges_of_their_tiles(dtype, H, P, N, G, taps, groups):
    """More state rows than 128 and columns than 64, sizes that fill a tile, sizes whose rows are no whole vectors, norms over runs of
    more than 1,024 and 2,048 channels."""
    test_state_space_kernels(dtype, H, P, N, G, taps, groups)


@pytest.mark.parametrize("far", [0, 1, 7, 8, 9, 63, 64, 65, 447, 511, 512])
def test_state_keeps_an_input_from_far_back(far):
    """With a decay of nearly 1 an input whose B matches the last token's C must come through from any distance: the first
    positions, the borders of the kernel's groups of tokens and of its chunks, hundreds of tokens back, also when the last token
    comes alone."""
    m = {"heads": 1, "vdim": 4, "state": 8, "groups": 1, "conv": 1, "norm_groups": 1}
    n, inner, N = 600, 4, 8
    g = torch.Generator().manual_seed(far)
    proj = 0.01 * torch.randn(n, 2 * inner + 2 * N + 1, generator=g)
    proj[:, :inner] = 5.0                                        # gate silu(5) ~ 5
    proj[:, -1] = 3.0                                            # dt ~ 3
    proj[far, inner: 2 * inner] = 9.0                            # x (silu(9) ~ 9)
    proj[far, 2 * inner + 3] = 9.0                               # B, state row 3
    proj[-1, 2 * inner + N + 3] = 9.0                            # C of the last token, state row 3
    ones, zeros = torch.ones(inner + 2 * N, 1), torch.zeros(inner + 2 * N)
    args = (m, ones, zeros, torch.zeros(1), torch.full((1,), -12.0), torch.zeros(1), torch.ones(inner), 1e-5)
    want = plain_state_space(proj, *args, [n])
    assert float(want[-1].abs().min()) > 0.9                      # the norm makes it 1: the far input dominates the last row
    for cuts, chunked in (((1.0,), False), ((1.0,), True), ((0.5, (n - 1) / n, 1.0), False), ((0.3, (n - 1) / n, 1.0), True)):
        got = run_state_space(proj, *args, torch.float32, [n], cuts, chunked)
        assert (got[-1].double() - want[-1]).abs().max() < 1e-3, (far, cuts, chunked)


# ------------------------------------------------------------------ the router, the experts' hidden units, pairs of tokens

@pytest.mark.parametrize("E,top,shared", [(5, 2, True), (3, 1, False), (7, 3, True), (2, 2, True), (64, 6, False)])
def test_routing_over_all_experts(E, top, shared):
    from pico_engine.ops import kernels
    g = torch.Generator().manual_seed(E)
    T, K = 50, 72
    x = torch.randn(T, K, generator=g)
    router = torch.randn(E, K, generator=g) * 0.5
    z = x.double() @ router.double().T
    s = torch.softmax(z, -1)
    want = torch.zeros(T, E + (1 if shared else 0), dtype=torch.float64)
    idx = s.topk(top, -1).indices
    want[:, :E].scatter_(1, idx, s.gather(1, idx) * 1.7)
    if shared:
        want[:, E] = 1.0
    extra = "one" if shared else False
    got = kernels.moe_route_stream(x.cuda(), None, 0.0, router.cuda().contiguous(), E, top, extra, over_all=True, factor=1.7)
    assert (got.cpu().double() - want).abs().max() < 1e-5
    got = kernels.moe_route(z.float().cuda().contiguous(), E, top, extra, over_all=True, factor=1.7)
    assert (got.cpu().double() - want).abs().max() < 1e-5
    # hidden units: relu^2 times the weight of the expert that owns the column; the shared expert's columns come last and may be wider
    # (widths that are multiples of 8 take 16-byte accesses in bfloat16); an infinite hidden unit behind a zero weight gives zero
    for ff, sff in ((12, 20), (16, 40)):
        h = torch.randn(T, E * ff + (sff if shared else 0), generator=g)
        unused = [e for e in range(E) if want[0, e] == 0]
        if unused:
            h[0, unused[0] * ff + 1] = float("inf")
        for dt, tol in ((torch.float32, 1e-5), (torch.bfloat16, 2e-2)):
            hh = h.to(dt)
            out = kernels.weighted_act(hh.cuda().contiguous(), "relu2", got, ff).float().cpu()
            col = torch.clamp(torch.arange(h.shape[1]) // ff, max=want.shape[1] - 1)
            w = want[:, col]
            ref = torch.where(w == 0, torch.zeros_like(w), plain.relu2(hh.double()) * w)
            assert (out.double() - ref).abs().max() < tol * float(ref.abs().max())
            assert bool((out[ref == 0] == 0).all())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_pairs_of_tokens_in_the_embedding(dtype):
    """Whole sequences, then the same cut into steps so that the token before comes from the state; slots are used again."""
    from pico_engine.ops import kernels
    dt = DTYPES[dtype]
    g = torch.Generator().manual_seed(5)
    V, W, buckets, mp, mc = 50, 24, 13, 29, 3
    table, pairs = torch.randn(V, W, generator=g).to(dt), torch.randn(buckets + 1, W, generator=g).to(dt)
    big = {"buckets": buckets, "mul_prev": mp, "mul_cur": mc}
    seqs = [torch.randint(0, V, (n,), generator=g).tolist() for n in (1, 7, 20)]
    w = {"embed": table.double(), "bigram": pairs.double()}
    want = [plain.embed(s, w, big) for s in seqs]
    state = torch.full((5, 1), 77, dtype=torch.int32).cuda()          # rows 0 and 4 belong to nobody
    for cuts in ([1.0], [0.5, 1.0], [0.2, 0.3, 0.9, 1.0]):
        done = [0] * len(seqs)
        got = [torch.zeros(len(s), W) for s in seqs]
        for c in cuts:
            upto = [len(s) if c == cuts[-1] else max(d, int(len(s) * c)) for s, d in zip(seqs, done)]
            rows = [b for b in range(len(seqs)) if upto[b] > done[b]]
            ids = torch.tensor([t for b in rows for t in seqs[b][done[b]:upto[b]]], dtype=torch.int32).cuda()
            lens = [upto[b] - done[b] for b in rows]
            pos = torch.tensor([p for b in rows for p in range(done[b], upto[b])], dtype=torch.int32).cuda()
            tr = torch.tensor(np.repeat(np.arange(len(rows)), lens), dtype=torch.int32).cuda()
            rf = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32).cuda()
            slots = torch.tensor([b + 1 for b in rows], dtype=torch.int32).cuda()
            out = kernels.embed_pairs(table.cuda(), pairs.cuda(), ids, pos, tr, rf, slots, state, buckets, mp, mc).cpu()
            at = 0
            for b, n in zip(rows, lens):
                got[b][done[b]:upto[b]] = out[at:at + n]; at += n
            done = upto
        for a, b in zip(got, want):
            assert (a.double() - b).abs().max() < 1e-6
        assert int(state[0, 0]) == 77 and int(state[4, 0]) == 77
        assert state[1:4, 0].tolist() == [s[-1] for s in seqs]


@pytest.mark.parametrize("rubbish", [float("nan"), float("inf")])
@pytest.mark.parametrize("H,width,rank", [(3, 96, 64), (2, 192, 128), (16, 256, 192)])
def test_prompts_over_low_rank_rows_do_not_see_what_an_earlier_owner_left_in_a_page(H, width, rank, rubbish):
    """Cache rows that no live sequence has written may hold anything: with numbers that are none in all of them, prompts that end on,
    before and behind the borders of pages and of runs give the same bits as with zeros."""
    from pico_engine.ops import kernels
    g = torch.Generator().manual_seed(width)
    for n, start in ((1, 0), (37, 0), (64, 0), (127, 0), (129, 0), (300, 0), (700, 650)):
        k, q = torch.randn(n, 1, width, generator=g), torch.randn(n - start, H * width, generator=g).bfloat16().cuda()
        got = []
        for fill in (0.0, rubbish):
            pool, table = paged(k, torch.bfloat16)
            pool[0] = fill
            if n % 64:
                pool[-1, :, n % 64:] = fill
            ctx = SimpleNamespace(one_token_each=False, scratch={}, lens=[n - start], starts=[start], dtype=torch.bfloat16)
            got.append(kernels.attention_latent_prompt(q, H * width, H, width, rank, pool, table, table.shape[1], None, width ** -0.5, ctx))
        kernels.check_status(torch.device("cuda", torch.cuda.current_device()))
        assert torch.equal(*got), (n, start)


@pytest.mark.parametrize("odd", [float("nan"), float("inf")])
@pytest.mark.parametrize("which", ["x", "B", "C"])
def test_a_token_that_is_no_number_does_not_reach_back(which, odd):
    """The state-space recurrence in chunks against the walk: what comes before the token is bit for bit what it is without it, and what
    comes behind is lost in the same places."""
    from pico_engine.ops import kernels
    H, P, N, G, lens = 2, 68, 32, 1, [130, 40]                                        # (no padding rows, whose zeros the walk multiplies too)
    g = torch.Generator().manual_seed(6)
    T, inner = sum(lens), H * P
    xbc, dt_raw = torch.randn(T, inner + 2 * G * N, generator=g), torch.randn(T, H, generator=g)
    first, rows, slots = (torch.tensor(v, dtype=torch.int32).cuda() for v in ([0, lens[0], T], lens, [0, 1]))

    def run(rows_in, chunked):
        state = torch.zeros(2, kernels.state_space_elems(H, P, N)).cuda()
        y = kernels.state_space_scan(rows_in.cuda(), dt_raw.cuda(), 0, torch.zeros(H).cuda(), torch.full((H,), -3.0).cuda(), torch.ones(H).cuda(),
                                     state, 0, first, rows, slots, H, P, N, G, chunked=chunked)
        return y.cpu(), state.cpu()

    clean = run(xbc, True)[0]
    column = {"x": 3, "B": inner + 1, "C": inner + G * N + 1}[which]
    for at in (5, 63, 100):
        bad = xbc.clone()
        bad[at, column] = odd
        (y, s), (y_walk, s_walk) = run(bad, True), run(bad, False)
        assert torch.equal(y[:at], clean[:at]) and torch.equal(y[lens[0]:], clean[lens[0]:]), at
        assert torch.equal(y.isfinite(), y_walk.isfinite()) and torch.equal(s.isfinite(), s_walk.isfinite()), at


def test_state_space_chunks_in_slabs():
    """More chunks than the scratch holds at once, sequences that end on, before and behind the borders of slabs: chunks against the walk."""
    from pico_engine.ops import kernels
    from pico_engine.ops.library import state_space
    H, P, N, G, lens = 64, 64, 128, 2, [3000, 64, 1, 65, 4999]
    T, B = sum(lens), len(lens)
    assert state_space().pe_state_space_slabs(T, B, H, P, N, G) > 1
    g = torch.Generator("cuda").manual_seed(2)
    xbc, dt_raw = torch.randn(T, H * P + 2 * G * N, generator=g, device="cuda"), torch.randn(T, H, generator=g, device="cuda")
    first, rows, slots = (torch.tensor(v, dtype=torch.int32).cuda() for v in (np.concatenate([[0], np.cumsum(lens)]), lens, range(B)))
    got = []
    for chunked in (False, True):
        state = torch.ones(B, kernels.state_space_elems(H, P, N), device="cuda")
        got.append((kernels.state_space_scan(xbc, dt_raw, 0, torch.full((H,), -3.0).cuda(), torch.linspace(-1, 1, H).cuda(), torch.ones(H).cuda(), state, 0,
                                             first, rows, slots, H, P, N, G, chunked=chunked), state))
    for walk, chunks in zip(*got):
        # float32 sums of the same products in another order (the bound of the tests above)
        assert (walk - chunks).abs().max() < 3e-5 * max(1.0, float(walk.abs().max()))


@pytest.mark.parametrize("H,width,rank", [(3, 256, 192), (2, 96, 64)])
def test_prompts_of_many_steps_over_low_rank_rows(monkeypatch, H, width, rank):
    """1,100 tokens, several rounds of the tcgen05 kernel's ring: one key that the last queries match, wherever it lies (the first
    positions, the borders of pages and of steps of 128 keys, late ones), and scores that rise from step to step, so that the outputs are
    rescaled every time."""
    from pico_engine.ops import kernels
    from pico_engine.ops.library import state_space
    assert state_space().pe_attention_latent_tcgen05_takes(width, rank)
    monkeypatch.setattr(kernels, "flashmix_prompts_pay", lambda *a: False)
    n, dt = 1100, torch.bfloat16
    g = torch.Generator().manual_seed(H)

    def check(q, k, window):
        i, j = torch.arange(n)[:, None], torch.arange(n)[None]
        seen = (j <= i) if window is None else (j <= i) & (i - j < window)
        w = torch.softmax(torch.einsum("ihd,jd->hij", q.double(), k[:, 0].double()).masked_fill(~seen, float("-inf")), -1)
        want = torch.einsum("hij,jd->ihd", w, k[:, 0, :rank].double())
        kp, table = paged(k, dt)
        got = run_attention(q, kp, None, table, dt, [(0, n)], window, 0, 1.0, None, rank, True)
        # weights and results are rounded to bfloat16, as in the tests above
        assert (got.double() - want).abs().max() < 2e-2 * max(1.0, float(want.abs().max()))
        return want

    noise = lambda *s: (0.02 * torch.randn(*s, generator=g)).to(dt).float()               # noqa: E731
    for far in (0, 63, 64, 127, 128, 511, 512, 767, 1000):
        q, k = noise(n, H, width), torch.randn(n, 1, width, generator=g).to(dt).float()
        k[:, :, rank:] = 0
        q[-5:] = 0
        q[-5:, :, -1] = k[far, :, -1] = 6.0
        k[far, :, :rank] = 8.0
        assert float(check(q, k, None)[-1].min()) > 7.9, far
    q, k = noise(n, H, width), torch.randn(n, 1, width, generator=g).to(dt).float()
    q[:, :, -1] = 2.0
    k[:, 0, -1] = (6.0 * torch.arange(n) / 128).to(dt).float()                             # 12 more with every 128 keys
    for window in (None, 200):
        check(q, k, window)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("taps,C,lens", [(4, 4608, [1, 2, 3, 127]), (2, 2048, [8, 9, 300]), (3, 4612, [5] * 44), (4, 5000, [1] * 70 + [2] * 69), (4, 1024, [1, 2, 127])])
def test_convolution_in_runs_of_channels(dtype, taps, C, lens):
    """Steps large enough for the kernel of four channels and eight tokens a thread (the last is not): rows that begin and end inside a thread's tokens, rows
    shorter than the taps, in two steps whose second reads what the first left."""
    from pico_engine.ops import kernels
    dt, B, T = DTYPES[dtype], len(lens), sum(lens)
    g = torch.Generator().manual_seed(C)
    w, bias = (0.5 * torch.randn(C, taps, generator=g)).to(dt), torch.randn(C, generator=g).to(dt)
    first, rows = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32).cuda(), torch.tensor(lens, dtype=torch.int32).cuda()
    tok_row = torch.tensor([b for b, n in enumerate(lens) for _ in range(n)], dtype=torch.int32).cuda()
    slots = torch.arange(B, dtype=torch.int32).flip(0).contiguous().cuda()
    state = torch.zeros(B, (taps - 1) * C).cuda()
    past = [torch.zeros(taps - 1, C, dtype=torch.float64) for _ in lens]
    for step in range(2):
        proj = torch.randn(T, C + 8, generator=g).to(dt)
        got = kernels.conv_silu(proj.cuda(), 4, C, w.cuda(), bias.cuda(), state, 0, tok_row, first, rows, slots).cpu().double()
        at = 0
        for b, n in enumerate(lens):
            u = torch.cat([past[b], proj[at: at + n, 4: 4 + C].double()])
            want = torch.nn.functional.silu(bias.double() + sum(w[:, j].double() * u[j: j + n] for j in range(taps)))
            # a sum of at most four products in float32, then silu
            assert (got[at: at + n] - want).abs().max() < 1e-5, (step, b)
            past[b], at = u[-(taps - 1):], at + n


def tensor_core_case(H, N, G, lens, seed, offset=0):
    """Inputs of the state-space recurrence at sizes whose prompts run on the tensor cores; rows that start ``offset`` numbers off a vector."""
    g = torch.Generator("cuda").manual_seed(seed)
    T, width = sum(lens), H * 64 + 2 * G * N
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    xbc = torch.empty(T * width + offset, device="cuda")[offset:].view(T, width)
    xbc.copy_(r(T, width))
    first, rows, slots = (torch.tensor(v, dtype=torch.int32).cuda() for v in (np.concatenate([[0], np.cumsum(lens)]), lens, range(len(lens))))
    steps = r(T, H), r(H) - 1.0, 0.7 * r(H) - 0.5, 1 + 0.3 * r(H)

    def run(rows_in, chunked, start=0.5):
        from pico_engine.ops import kernels
        state = torch.full((len(lens), kernels.state_space_elems(H, 64, N)), start, device="cuda")
        y = kernels.state_space_scan(rows_in, steps[0], 0, *steps[1:], state, 0, first, rows, slots, H, 64, N, G, chunked=chunked)
        kernels.check_status(torch.device("cuda", torch.cuda.current_device()))
        return y, state
    return xbc, run


@pytest.mark.parametrize("H,N,G,offset", [(2, 64, 1, 0), (2, 128, 1, 0), (12, 128, 2, 1), (10, 64, 5, 0), (6, 64, 3, 3)])
def test_state_space_products_on_the_tensor_cores(H, N, G, offset):
    """Chunks that end on, before and behind their 64 tokens, more units than blocks, rows off a vector: products in bfloat16 parts against the walk."""
    lens = [1, 63, 64, 65, 128, 1000, 700, 7] + [64] * (40 if H > 6 else 1)
    xbc, run = tensor_core_case(H, N, G, lens, H + N, offset)
    for walk, chunks in zip(run(xbc, False), run(xbc, True)):
        # float32 sums of the same products in another order (the bound of the tests above)
        assert (walk - chunks).abs().max() < 3e-5 * max(1.0, float(walk.abs().max()))


@pytest.mark.parametrize("odd", [float("nan"), float("-inf"), 3.4e38])
@pytest.mark.parametrize("N,which", [(64, "x"), (128, "B"), (128, "C")])
def test_numbers_that_parts_do_not_hold_stay_where_they_are(odd, N, which):
    """A number that is none, an infinity, and one that rounds to an infinity: tokens in front keep their bits, and the places that are lost are the walk's."""
    H, G, lens = 4, 2, [130, 40]
    xbc, run = tensor_core_case(H, N, G, lens, N)
    clean = run(xbc, True)[0]
    column = {"x": 70, "B": H * 64 + 1, "C": H * 64 + G * N + 1}[which]
    for at in (0, 5, 63, 100):
        bad = xbc.clone()
        bad[at, column] = odd
        (y, s), (y_walk, s_walk) = run(bad, True), run(bad, False)
        assert torch.equal(y[:at], clean[:at]) and torch.equal(y[lens[0]:], clean[lens[0]:]), at
        if odd != 3.4e38:                                     # (products of it may or may not leave float32, by their order)
            assert torch.equal(y.isfinite(), y_walk.isfinite()) and torch.equal(s.isfinite(), s_walk.isfinite()), at


@pytest.mark.parametrize("scale", [1e-36, 1e-30, 1e30])
def test_state_space_products_at_the_ends_of_the_range(scale):
    """x far below and far above one: errors as large, beside the results, as at one (numbers of 2^35 and more are multiplied as they are)."""
    xbc, run = tensor_core_case(4, 128, 2, [200], 3)
    xbc[:, :256] *= scale
    walk, chunks = run(xbc, False)[0], run(xbc, True)[0]
    # the state begins at 0.5: at 1e-36 nothing of x is left beside it
    assert (walk - chunks).abs().max() < 3e-5 * float(walk.abs().max())


@pytest.mark.parametrize("H,N,G,lens,most_y,most_state", [(8, 64, 1, [65, 1], 5.7e-8, 9.6e-8), (28, 64, 2, [300, 100], 6.3e-8, 1.04e-7), (28, 128, 2, [300, 100], 1.04e-7, 1.06e-7)])
def test_state_space_errors_are_no_larger_than_multiply_adds(H, N, G, lens, most_y, most_state):
    """Outputs and states against 64 bits, beside their norms, means over eight inputs; the bounds are what the multiply-add tiles leave of such inputs."""
    from pico_engine.ops import kernels
    errors = []
    for seed in range(8):
        g = torch.Generator("cuda").manual_seed(seed)
        r = lambda *s: torch.randn(*s, device="cuda", generator=g)                       # noqa: E731
        T, split = sum(lens), kernels.state_space_split(N)
        xbc, dt_raw = torch.nn.functional.silu(r(T, H * 64 + 2 * G * N)), r(T, H)
        dt0 = torch.exp(torch.rand(H, device="cuda", generator=g) * 4.6 - 6.9)           # steps of 0.001 to 0.1, decay rates of 1 to 16
        bias, a_log, skip = dt0 + torch.log(-torch.expm1(-dt0)), torch.log(1 + 15 * torch.rand(H, device="cuda", generator=g)), 1 + 0.05 * r(H)
        first, rows, slots = (torch.tensor(v, dtype=torch.int32).cuda() for v in (np.concatenate([[0], np.cumsum(lens)]), lens, range(len(lens))))
        state = torch.zeros(len(lens), kernels.state_space_elems(H, 64, N), device="cuda")
        y = kernels.state_space_scan(xbc, dt_raw, 0, bias, a_log, skip, state, 0, first, rows, slots, H, 64, N, G, chunked=True)
        got = state.view(len(lens), H, N // split, 64, split).permute(0, 1, 4, 2, 3).reshape(len(lens), H, N, 64)
        x, b, c = (t.double() for t in xbc.split([H * 64, G * N, G * N], 1))
        x, (b, c) = x.view(T, H, 64), (t.view(T, G, N).repeat_interleave(H // G, 1) for t in (b, c))
        dt = torch.nn.functional.softplus(dt_raw.double() + bias.double(), threshold=100.0)
        decay, want, ends, at = torch.exp(-torch.exp(a_log.double()) * dt), torch.empty_like(x), [], 0
        for n in lens:
            S = torch.zeros(H, N, 64, dtype=torch.float64, device="cuda")
            for t in range(at, at + n):
                S = decay[t][:, None, None] * S + (dt[t][:, None] * b[t])[:, :, None] * x[t][:, None]
                want[t] = (c[t][:, None] @ S)[:, 0] + skip.double()[:, None] * x[t]
            ends.append(S)
            at += n
        ends = torch.stack(ends)
        errors.append([float((y.view(T, H, 64) - want).norm() / want.norm()), float((got - ends).norm() / ends.norm())])
    e_y, e_state = np.mean(errors, 0)
    assert e_y < most_y and e_state < most_state, (e_y, e_state)


@pytest.mark.parametrize("what", ["a head", "a column", "B", "C", "all"])
@pytest.mark.parametrize("N", [64, 128])
def test_tiny_numbers_beside_others_keep_their_digits(N, what):
    """One head's x, one column of it, a token's B or C, and everything, 2^-122 beside numbers near one: each result to float32 of its own size."""
    H, G, lens, tiny = 4, 2, [200, 65], 2.0 ** -122
    xbc, run = tensor_core_case(H, N, G, lens, 7)
    inner = H * 64
    if what == "a head":
        xbc[:, 64:128] *= tiny
    elif what == "a column":
        xbc[:, 130] *= tiny
    elif what == "B":
        xbc[:, inner: inner + G * N] *= tiny
    elif what == "C":
        xbc[70, inner + G * N:] *= tiny
        xbc[70, :inner] = 0.0                                 # (the token's own x joins its output as it is)
    else:
        xbc[:, :inner] *= tiny
    for walk, chunks in zip(run(xbc, False, 0.0), run(xbc, True, 0.0)):
        if walk.shape[0] == len(lens):                        # states: [sequence][head][rows and columns]
            walk, chunks = (s.view(len(lens), H, -1) for s in (walk, chunks))
        else:                                                 # outputs: a column a result of its own
            walk, chunks = (y.view(-1, H, 64).permute(0, 1, 2) for y in (walk, chunks))
            rows = [70] if what == "C" else list(range(65))   # (from the first sequence: the second begins anew)
            walk, chunks = walk[rows], chunks[rows]
            if what == "a column":
                walk, chunks = walk[:, :, 2:3], chunks[:, :, 2:3]
        # float32 sums of the same products in another order, beside the largest of the head (the bound of the tests above)
        size = walk.abs().amax(dim=(0, 2), keepdim=True)
        assert ((walk - chunks).abs() <= 3e-5 * size).all()


@pytest.mark.parametrize("T", [1, 3, 130])
@pytest.mark.parametrize("H,D,R,rank,rot,rows,absorbed", [(1, 8, 8, 8, 8, False, True), (16, 128, 64, 192, 64, False, False), (5, 16, 24, 256, 16, True, True), (3, 8, 16, 40, 0, False, True),
                                                          (60, 8, 64, 64, 64, True, False)])
def test_low_rank_rows_in_runs_of_eight(T, H, D, R, rank, rot, rows, absorbed):
    """The kernel that takes eight entries a thread against the general one, which takes the same numbers from a place one entry further on."""
    from pico_engine.ops import kernels
    g = torch.Generator("cuda").manual_seed(rank + T)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    width, W = H * (D + R), rank + R
    proj, q_rows, qa, weight = r(T, width + W), r(T, width) if rows else None, r(H, T, rank) if absorbed else None, 1 + 0.1 * r(rank)
    freq = 10000.0 ** (-torch.arange(max(rot // 2, 1), device="cuda") / max(rot // 2, 1))
    pos = torch.randperm(5000, generator=g, device="cuda")[:T].int().sort().values       # (no place of the cache twice)
    pages = int(pos.max()) // 64 + 1
    table = torch.randperm(pages, generator=g, device="cuda").int().view(1, pages)
    got = []
    for shift in (0, 1):
        put = lambda t: None if t is None else torch.empty(t.numel() + shift, dtype=t.dtype, device="cuda")[shift:].view(t.shape).copy_(t)
        pool, out = torch.zeros(pages, 1, 64, W, dtype=torch.bfloat16, device="cuda"), torch.zeros(T, H * W, dtype=torch.bfloat16, device="cuda")
        q = kernels.latent_prepare(put(proj), H, D, R, rank, width, weight, 1e-5, freq, rot, put(qa), pos, torch.zeros(T, dtype=torch.int32, device="cuda"), pool, table, pages,
                                   q_rows=put(q_rows), q_out=None if absorbed else out)
        got.append((q.float(), pool.float()))
    for a, b in zip(*got):                                     # the same arithmetic in the same order
        assert torch.equal(a, b)


@pytest.mark.parametrize("which", ["x", "B"])
def test_a_sequence_that_is_no_number_does_not_hold_up_the_others(which):
    """A batch's step with one such sequence takes about as long as without it: 1.3 to 1.5 times where a walk from memory took 5 to 9."""
    xbc, run = tensor_core_case(64, 128, 2, [1400, 647], 2)
    bad = xbc.clone()
    bad[5, 3 if which == "x" else 64 * 64 + 3] = float("nan")

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
    assert time(bad) < 3 * time(xbc)
