"""The engine's host logic (packing, paging, rings, slots, schedules) on a machine without a GPU:
the CUDA entry points are replaced by the plain functions of tests/kernel_refs.py, everything
above them is the product's code.  Logits are compared with the plain implementation."""
import os

import numpy as np
import pytest
import torch

import kernel_refs
import plain_gemma2 as plain
import tiny_configs
from rust_deeplearning_b200.config.base import architecture_for
from rust_deeplearning_b200.engine.step import Engine
from rust_deeplearning_b200.kernels import library
from rust_deeplearning_b200.parts.model import Model
from rust_deeplearning_b200.weights.loader import load_weights
from rust_deeplearning_b200.weights.random_init import write_random_model

TOL = 2e-5   # float32 activations between float64 kernels


def build(tmp_path, name, monkeypatch, page_size=4, max_tokens=4096, max_seqs=None):
    kernel_refs.install(monkeypatch)
    cfg, seed = tiny_configs.config(name)
    folder = str(tmp_path / f"tiny_{name}")
    write_random_model(folder, cfg, seed, "float32")
    arch = architecture_for(cfg)
    spec = arch.build_spec(arch.parse_config(cfg))
    model = Model(spec, load_weights(spec, folder, torch.float32, "cpu"), torch.float32, "cpu")
    engine = Engine(model, max_tokens=max_tokens, max_seqs=max_seqs, page_size=page_size, use_graphs=False)
    pcfg, pw = plain.load_folder(folder)
    return engine, pcfg, pw


def prompt(rng, n, vocab):
    return [int(v) for v in rng.integers(0, vocab, size=n)]


def close(got, want):
    got = got.detach().cpu().double().numpy()
    assert got.shape == want.shape
    assert np.isfinite(got).all()
    assert np.abs(got - want).max() <= TOL, np.abs(got - want).max()


@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_whole_prompt_equals_plain(tmp_path, monkeypatch, name):
    engine, cfg, w = build(tmp_path, name, monkeypatch)
    rng = np.random.default_rng(1)
    ids = prompt(rng, 37, cfg["vocab_size"])          # longer than both windows
    slot = engine.new_sequence()
    logits = engine.step([slot], [ids], "all")
    close(logits, plain.forward(cfg, w, ids))


@pytest.mark.parametrize("name", ["A", "B"])
def test_token_by_token_and_chunks_equal_plain(tmp_path, monkeypatch, name):
    engine, cfg, w = build(tmp_path, name, monkeypatch)
    rng = np.random.default_rng(2)
    ids = prompt(rng, 45, cfg["vocab_size"])
    want = plain.forward(cfg, w, ids)
    # a prefix whole, then one by one
    slot = engine.new_sequence()
    close(engine.step([slot], [ids[:13]], "all"), want[:13])
    for t in range(13, 45):
        close(engine.step([slot], [[ids[t]]], "all"), want[t:t + 1])
    engine.release(slot)
    # the same in three chunks: a chunk after an existing prefix reads cache and new rows
    slot = engine.new_sequence()
    close(engine.step([slot], [ids[:7]], "all"), want[:7])
    close(engine.step([slot], [ids[7:30]], "all"), want[7:30])
    close(engine.step([slot], [ids[30:]], "all"), want[30:])


@pytest.mark.parametrize("name", ["A", "B"])
def test_unequal_batches_and_slot_reuse(tmp_path, monkeypatch, name):
    engine, cfg, w = build(tmp_path, name, monkeypatch, max_tokens=256, max_seqs=4)
    rng = np.random.default_rng(3)
    V = cfg["vocab_size"]
    for round_ in range(3):                      # one batch after another on the same small cache
        lens = [1, 9, 23, 40] if round_ % 2 == 0 else [17, 5, 11]
        extra = [3, 12, 6, 1]
        seqs = [prompt(rng, n + e, V) for n, e in zip(lens, extra)]
        want = [plain.forward(cfg, w, s) for s in seqs]
        slots = [engine.new_sequence() for _ in seqs]
        got = engine.step(slots, [s[:n] for s, n in zip(seqs, lens)], "all")
        close(got, np.concatenate([wv[:n] for wv, n in zip(want, lens)]))
        pos = list(lens)
        live = list(range(len(seqs)))
        while live:
            got = engine.step([slots[i] for i in live], [[seqs[i][pos[i]]] for i in live], "last")
            close(got, np.stack([want[i][pos[i]] for i in live]))
            for i in live:
                pos[i] += 1
            for i in [i for i in live if pos[i] == len(seqs[i])]:
                engine.release(slots[i])         # shorter requests end earlier
            live = [i for i in live if pos[i] < len(seqs[i])]
        assert engine.cache.n_free_slots == 4
        assert all(g.pool.n_free == g.pool.n_pages for g in engine.cache.kv_groups)


def test_wanted_places_and_errors(tmp_path, monkeypatch):
    engine, cfg, w = build(tmp_path, "A", monkeypatch)
    from rust_deeplearning_b200.engine.step import StepError
    rng = np.random.default_rng(4)
    a, b = prompt(rng, 6, 256), prompt(rng, 11, 256)
    s0, s1 = engine.new_sequence(), engine.new_sequence()
    got = engine.step([s0, s1], [a, b], [[0, 5], []])
    close(got, plain.forward(cfg, w, a)[[0, 5]])
    assert engine.length(s0) == 6 and engine.length(s1) == 11
    got = engine.step([s1, s0], [[3], [4]], [[0], []])
    close(got, plain.forward(cfg, w, b + [3])[-1:])
    with pytest.raises(StepError):
        engine.step([s0], [[256]])
    with pytest.raises(StepError):
        engine.step([s0], [[]])
    with pytest.raises(StepError):
        engine.step([s0], [[1.5]])                # no whole number: refused, not cut down to 1
    with pytest.raises(StepError):
        engine.step([s0], [[True]])
    with pytest.raises(StepError):
        engine.step([s0], [[3, 4]], [[0.5]])
    assert engine.length(s0) == 7                 # failed steps changed nothing


def test_a_walk_of_valid_and_invalid_steps_drawn_at_random(tmp_path, monkeypatch):
    """Four slots on a cache of 160 rows: sequences begin and are given back, steps bring 1 to 17 tokens for any
    subset of them and want any places, and about a third of the steps are wrong in one way (an empty list, an id
    outside the vocabulary or no whole number, a slot twice or not in use, a wanted place outside, more tokens than
    the context or the cache holds, tokens for too few sequences).  A wrong step raises the engine's own error and
    changes no length; a right one gives the plain implementation's logits, whatever came before."""
    import random
    from rust_deeplearning_b200.cache.cache import CacheError
    from rust_deeplearning_b200.engine.step import StepError
    engine, cfg, w = build(tmp_path, "A", monkeypatch, page_size=4, max_tokens=160, max_seqs=4)
    V = cfg["vocab_size"]
    rnd = random.Random(5)
    live, checked, refused = {}, 0, 0          # slot -> the tokens it holds
    for _ in range(90):
        kind = rnd.random()
        if kind < 0.15 and len(live) < 4:
            live[engine.new_sequence()] = []
            continue
        if kind < 0.25 and live:
            slot = rnd.choice(list(live))
            engine.release(slot)
            del live[slot]
            continue
        if kind < 0.30:
            with pytest.raises((StepError, CacheError)):
                if rnd.random() < 0.5:
                    engine.release(rnd.choice([-1, 99] + [s for s in range(4) if s not in live]))
                else:
                    for _ in range(5 - len(live)):
                        live[engine.new_sequence()] = []
            refused += 1
            continue
        if not live:
            continue
        slots = rnd.sample(list(live), rnd.randint(1, len(live)))
        toks = [[rnd.randrange(V) for _ in range(rnd.choice([1, 1, 2, 5, 17]))] for _ in slots]
        want = rnd.choice(["last", "all", None])
        if want is None:
            want = [sorted(rnd.sample(range(len(t)), rnd.randint(0, len(t)))) for t in toks]
        before = {s: engine.length(s) for s in live}
        if rnd.random() < 0.35:
            k = rnd.randrange(9)
            if k == 0: toks[0] = []
            elif k == 1: toks[0] = [V + rnd.randrange(3)]
            elif k == 2: toks[0] = [-1]
            elif k == 3: slots, toks = slots + [slots[0]], toks + [toks[0]]
            elif k == 4: slots[0] = rnd.choice([-1, 99] + [s for s in range(4) if s not in live])
            elif k == 5: want = [[len(t)] for t in toks]
            elif k == 6: toks[0] = [rnd.randrange(V) for _ in range(600)]
            elif k == 7: toks = toks[:-1] if len(toks) > 1 else toks + [[1]]
            elif k == 8: toks[0] = [1.5]
            if k in (5, 7) and not isinstance(want, str) and len(want) != len(toks):
                want = "last"
            with pytest.raises((StepError, CacheError)):
                engine.step(slots, toks, want)
            assert {s: engine.length(s) for s in live} == before, f"a refused step (kind {k}) changed a length"
            refused += 1
            continue
        try:
            got = engine.step(slots, toks, want)
        except CacheError:                      # the cache is full: nothing may have changed
            assert {s: engine.length(s) for s in live} == before
            refused += 1
            continue
        places = [[len(t) - 1] for t in toks] if want == "last" else ([list(range(len(t))) for t in toks] if want == "all" else want)
        rows = []
        for slot, t, ws in zip(slots, toks, places):
            if ws:
                rows += list(plain.forward(cfg, w, live[slot] + t)[[len(live[slot]) + i for i in ws]])
            live[slot] = live[slot] + t
        if rows:
            close(got, np.stack(rows))
            checked += 1
    assert checked > 20 and refused > 10, (checked, refused)


def test_a_run_that_reads_another_runs_ring_sees_the_rows_of_earlier_steps(tmp_path, monkeypatch):
    """Schedule: layer 0 with a window of 8 keeps a ring of 3 pages of 4 rows; layer 1 reads layer 0's keys and
    values.  A portion of 10 tokens on a prefix of 9 lands on ring rows that the portion's early queries still
    read in layer 1, so layer 0's write has to wait until layer 1 has run.  Whole, in portions and token by
    token must agree (the whole prompt reads no ring at all)."""
    import dataclasses
    from rust_deeplearning_b200.parts.spec import ScheduleEntry
    kernel_refs.install(monkeypatch)
    cfg, seed = tiny_configs.config("A")
    cfg["layer_types"] = ["sliding_attention", "sliding_attention"]
    folder = str(tmp_path / "shared")
    write_random_model(folder, cfg, seed, "float32")
    arch = architecture_for(cfg)
    spec = arch.build_spec(arch.parse_config(cfg))
    spec = dataclasses.replace(spec, schedule=(ScheduleEntry(0), ScheduleEntry(1, reads_cache_of=0)))
    model = Model(spec, load_weights(spec, folder, torch.float32, "cpu"), torch.float32, "cpu")
    engine = Engine(model, max_tokens=4096, page_size=4, use_graphs=False)
    assert engine.cache.kv_groups[0].is_ring and engine.cache.kv_groups[0].ring_pages == 3
    rng = np.random.default_rng(9)
    ids = prompt(rng, 40, cfg["vocab_size"])
    slot = engine.new_sequence()
    whole = engine.step([slot], [ids], "all").double().numpy()
    engine.release(slot)
    slot = engine.new_sequence()
    parts = [engine.step([slot], [ids[a:b]], "all") for a, b in ((0, 9), (9, 19), (19, 20), (20, 40))]
    close(torch.cat(parts), whole)
    engine.release(slot)
    slot = engine.new_sequence()
    close(torch.cat([engine.step([slot], [[t]], "all") for t in ids]), whole)


def test_prompt_attention_blocks_follow_the_keys_and_the_room():
    """How many blocks share a query tile and head: no more than a short prompt's keys can feed, no more than find room at once
    (two a multiprocessor where their memory allows; clusters of four and eight leave an eighth of them empty)."""
    from rust_deeplearning_b200.kernels import library
    blocks = lambda pairs, hd, keys, sigmoid=0: library.load().rdl_attention_prefill_blocks(pairs, hd, sigmoid, keys, 148)
    assert [blocks(8, 256, k) for k in (0, 1, 64, 256, 257, 8000)] == [8, 4, 4, 4, 8, 8]           # (0: not known)
    assert [blocks(p, 256, 700) for p in (1, 32, 33, 64, 65, 148, 149, 10 ** 9)] == [8, 8, 4, 4, 2, 2, 1, 1]
    assert [blocks(p, 256, 700, 1) for p in (16, 17, 32, 33, 74, 75)] == [8, 4, 4, 2, 2, 1]        # its memory leaves room for one
    assert [blocks(p, 64, 700) for p in (32, 64, 65, 148)] == [8, 4, 1, 1]
    assert [blocks(p, 16, 45) for p in (64, 65)] == [4, 1]


def test_delta_rule_columns_follow_the_walk(tmp_path, monkeypatch):
    """Two columns a lane where the tokens fill the chip beside the longest sequence, not where sequences of a few tokens stand beside it;
    the engine says how long the longest is."""
    columns = lambda lens, heads=16, vdim=128: library.load().rdl_delta_rule_columns(sum(lens), len(lens), max(lens), heads, vdim, 148)
    assert [columns(x) for x in ([1500], [700] * 2, [1500, 10, 10], [1500] + [10] * 7, [10] * 7 + [1500], [1500, 600, 300])] == [1] * 6
    assert [columns(x) for x in ([1000] * 3, [400] * 4, [60] * 64, [200, 633, 1066, 1500], [1500, 1000, 500], [800] + [100] * 16)] == [2] * 6
    assert [columns([n] * 9, 2, 256) for n in (1, 10 ** 6)] == [1, 1] and [columns([n] * 10, 2, 256) for n in (1, 10 ** 6)] == [2, 2]
    assert [columns([1500] + [10] * n, vdim=64) for n in (3, 4)] == [1, 2]          # its own blocks take less than half of the chip
    assert library.load().rdl_delta_rule_columns(1570, 8, 0, 16, 128, 148) == 2     # not known
    engine, _, _ = build(tmp_path, "A", monkeypatch)
    seen, forward = [], engine._forward
    monkeypatch.setattr(engine, "_forward", lambda batch: seen.append(batch.longest_new) or forward(batch))
    engine.step([engine.new_sequence() for _ in range(3)], [[1, 2], [3] * 9, [4]])
    assert seen == [9]


def test_tiles_of_the_32_bit_product_follow_the_waves():
    """Rows of a tile, chunks of the ring, and whether eight blocks share a tile, on 148 multiprocessors: short tiles where all find room
    at once, tall ones where fewer waves do; no ring that leaves room for fewer clusters than the tiles need."""
    form = lambda m, n, k=4096, sms=148: library.load().rdl_gemm_f32_form(m, n, k, sms)
    assert [form(m, 256) for m in (1, 16, 17, 64, 96)] == [0, 0, 3221, 3221, 3221]
    assert [form(m, 1000) for m in (96, 128)] == [3221, 3231]                      # 16 clusters of one block a multiprocessor do not find room
    assert [form(m, 2304) for m in (32, 48, 64, 96, 128, 200)] == [3221, 4821, 3221, 4821, 3221, 4821]
    assert [form(m, 4096) for m in (32, 48, 64, 128, 512)] == [3231, 4831, 6421, 6421, 12830]
    assert [form(m, 3584) for m in (112, 128, 512)] == [12831, 12831, 4821]
    assert [form(m, 18432) for m in (48, 64, 128)] == [4821, 6421, 12830]
    assert [form(m, 8000, 300) for m in (400, 800)] == [6420, 12830]               # short sums: the meetings of shared tiles weigh more
    assert [form(48, 128 * n) // 10 % 10 for n in (24, 25, 33, 34)] == [2, 3, 3, 2]
    for m in (17, 32, 33, 64, 97, 300, 5000, 65535 * 48 + 1, 65535 * 64):
        for n in (1, 128, 129, 5000, 300000):
            for sms in (1, 8, 132, 148):
                rows, rest = divmod(form(m, n, 4096, sms), 100)
                assert rows in (32, 48, 64, 128) and rest in (20, 21, 30, 31) and -(-m // rows) <= 65535, (m, n, sms)


def test_no_launch_reads_the_environment():
    """A launcher runs on every step: what the environment may set is read once, into a static."""
    folder = os.path.dirname(os.path.abspath(library.__file__)) + "/../csrc/"
    for f in sorted(os.listdir(folder)):
        with open(folder + f, encoding="utf-8") as fh:
            for line in fh:
                assert "getenv" not in line or line.strip().startswith("static const"), (f, line)


def test_what_a_device_needs_raised_is_raised_on_every_device(tmp_path):
    """`csrc/per_device.h`, which the launchers keep the opt-in to more shared memory with: asked for once a device and size, again
    where it failed, never lowered, and by several threads."""
    import os
    import shutil
    import subprocess
    from rust_deeplearning_b200.kernels import library
    src = tmp_path / "t.cpp"
    src.write_text(r"""
#include "per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
int main() {
    RdlRaisedPerDevice r;
    int calls = 0, result = 0;
    auto f = [&] { ++calls; return result; };
    auto want = [&](int device, int value, int status, int n, int line) {
        calls = 0;
        const int e = r.run(device, value, f);
        if (e != status || calls != n) { std::printf("line %d: %d, %d calls\n", line, e, calls); std::exit(1); }
    };
    want(0, 100, 0, 1, __LINE__);
    want(0, 100, 0, 0, __LINE__);
    want(1, 100, 0, 1, __LINE__);      // another device has not been asked
    want(0, 50, 0, 0, __LINE__);
    want(0, 200, 0, 1, __LINE__);
    want(1, 100, 0, 0, __LINE__);
    result = 7;
    want(63, 10, 7, 1, __LINE__);
    want(63, 10, 7, 1, __LINE__);      // a failure is not remembered
    result = 0;
    want(63, 10, 0, 1, __LINE__);
    want(64, 10, 0, 1, __LINE__);
    want(64, 10, 0, 1, __LINE__);
    int set = 0;                       // threads with other sizes: the last one set is the largest
    std::vector<std::thread> ts;
    for (int t = 1; t <= 8; ++t) ts.emplace_back([&, t] { for (int i = 0; i < 1000; ++i) r.run(5, t * 1000 + i, [&] { set = t * 1000 + i; return 0; }); });
    for (auto& t : ts) t.join();
    if (set != 8999) { std::printf("ended at %d\n", set); return 1; }
    return 0;
}
""")
    exe = tmp_path / "t"
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-O1", "-pthread", "-I", library.CSRC, "-include", "cstdlib", str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
    for name in os.listdir(library.CSRC):       # nobody keeps such a thing once a process
        text = open(os.path.join(library.CSRC, name)).read()
        assert name == "launch.cuh" or "cudaFuncSetAttribute" not in text, name
