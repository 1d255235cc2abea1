"""Generation through the entry point: greedy and sampled, graph-replayed and plain, against the
plain implementation; stop tokens, sequences that end earlier, batches one after another."""
import numpy as np
import pytest
import torch

import plain_llama
from helpers import TINY, make_model_dir, random_tokens

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    out = {}
    for which, (cfg_dict, seed) in TINY.items():
        d = make_model_dir(tmp_path_factory.mktemp(f"gen_{which}"), cfg_dict, seed, torch.bfloat16)
        out[which] = (d,) + plain_llama.read_model_folder(d)
    return out


@pytest.mark.parametrize("use_graphs", [False, True])
@pytest.mark.parametrize("which,lens", [("a", [5, 9, 1]), ("b", [17, 3, 40, 11])])
def test_greedy_float32_matches_plain(models, which, lens, use_graphs):
    from fastgguf_b200.engine.api import Engine
    model_dir, cfg, W = models[which]
    prompts = [random_tokens(n, cfg["vocab_size"], 50 + i) for i, n in enumerate(lens)]
    engine = Engine.from_dir(model_dir, dtype="float32", max_tokens=1024, max_batch=4, use_graphs=use_graphs)
    out = engine.generate(prompts, temp=0, max_tokens=8, ignore_eos=True)
    for p, c in zip(prompts, out):
        want = plain_llama.plain_generate(cfg, W, p, max_tokens=8, temp=0, top_k=0, top_p=1.0, repeat_penalty=1.0,
                                          repeat_last_n=64)
        assert c.tokens == want and c.finish_reason == "length"
    engine.cache.check()
    assert engine.cache.live_slots() == []


@pytest.mark.parametrize("use_graphs", [False, True])
def test_sampled_float32_matches_plain(models, use_graphs):
    """Temperature 0.8 with the reference's default top-k / top-p, and a repeat penalty: same logits,
    same generator state, same token - also for the second batch, whose slots were used before."""
    from fastgguf_b200.engine.api import Engine
    from fastgguf_b200.sampling import request_seed
    model_dir, cfg, W = models["b"]
    prompts = [random_tokens(n, cfg["vocab_size"], 60 + i) for i, n in enumerate([17, 3, 40, 11, 6])]
    engine = Engine.from_dir(model_dir, dtype="float32", max_tokens=1024, max_batch=4, use_graphs=use_graphs)
    opts = dict(temp=0.8, top_k=64, top_p=0.95, repeat_penalty=1.3, repeat_last_n=16)
    out = engine.generate(prompts, max_tokens=12, seed=7, ignore_eos=True, batch_size=3, **opts)
    for i, (p, c) in enumerate(zip(prompts, out)):
        want = plain_llama.plain_generate(cfg, W, p, max_tokens=12, seed=request_seed(7, i), **opts)
        assert c.tokens == want, i


@pytest.mark.parametrize("use_graphs", [False, True])
def test_stop_tokens_and_early_finish(models, use_graphs):
    """A stop token ends its sequence without being emitted; the others go on; slots come back."""
    from fastgguf_b200.engine.api import Engine
    model_dir, cfg, W = models["a"]
    prompts = [random_tokens(n, cfg["vocab_size"], 70 + i) for i, n in enumerate([4, 12, 7, 2, 9])]
    free = [plain_llama.plain_generate(cfg, W, p, max_tokens=10, temp=0, top_k=0, top_p=1.0, repeat_penalty=1.0,
                                       repeat_last_n=64) for p in prompts]
    stops = {free[0][3], free[2][0]}               # sequence 0 stops before its 4th token, sequence 2 at once
    want = []
    for toks in free:
        cut = next((k for k, t in enumerate(toks) if t in stops), None)
        want.append((toks if cut is None else toks[:cut], "length" if cut is None else "stop"))
    engine = Engine.from_dir(model_dir, dtype="float32", max_tokens=512, max_batch=2, use_graphs=use_graphs)
    out = engine.generate(prompts, temp=0, max_tokens=10, stop_ids=sorted(stops), batch_size=2)
    assert [(c.tokens, c.finish_reason) for c in out] == want
    engine.cache.check()
    assert engine.cache.live_slots() == []


def test_greedy_bfloat16_is_plausible(models):
    """bfloat16 greedy tokens: each chosen token's float64 logit lies within rounding of the maximum."""
    from fastgguf_b200.engine.api import Engine
    model_dir, cfg, W = models["b"]
    prompts = [random_tokens(n, cfg["vocab_size"], 80 + i) for i, n in enumerate([20, 5, 33])]
    engine = Engine.from_dir(model_dir, dtype="bfloat16", max_tokens=1024, max_batch=4)
    out = engine.generate(prompts, temp=0, max_tokens=16, ignore_eos=True)
    for p, c in zip(prompts, out):
        assert len(c.tokens) == 16
        logits = plain_llama.plain_forward(cfg, W, p + c.tokens).numpy()
        for k, tok in enumerate(c.tokens):
            row = logits[len(p) - 1 + k]
            assert row[tok] >= row.max() - 3e-2 * np.abs(row).max()


def test_context_full_ends_with_length(models):
    from fastgguf_b200.engine.api import Engine
    model_dir, cfg, W = models["a"]
    engine = Engine.from_dir(model_dir, dtype="float32", max_tokens=256, max_batch=2, max_seq_len=64)
    out = engine.generate([random_tokens(60, cfg["vocab_size"], 90)], temp=0, max_tokens=0, ignore_eos=True)
    # 60 prompt tokens + 4 fed tokens fill the 64 positions; the 5th sampled token is still emitted
    assert len(out[0].tokens) == 5 and out[0].finish_reason == "length"


def test_calls_that_differ_only_in_seed_share_one_backend_and_few_option_sets_are_kept(models):
    """The recorded decode graphs belong to a set of sampling options, not to a seed: new seeds record nothing, and of
    many option sets only the most recent few keep their graphs and activation memory."""
    from fastgguf_b200.engine.api import Engine
    d, cfg, _ = models["a"]
    engine = Engine.from_dir(d, dtype="bfloat16", max_tokens=1024, max_batch=2)
    prompts = [[3, 5, 7, 11], [2, 4]]
    engine.generate(prompts, max_tokens=4, temp=0.9, top_k=8, top_p=0.9, seed=1, ignore_eos=True)
    first = engine.stats()
    assert first["backends"] == 1 and first["graphs"] >= 1
    outs = [engine.generate(prompts, max_tokens=4, temp=0.9, top_k=8, top_p=0.9, seed=s, ignore_eos=True) for s in (2, 3, 2)]
    after = engine.stats()
    assert after["backends"] == 1 and after["graphs"] == first["graphs"]
    assert [c.tokens for c in outs[0]] == [c.tokens for c in outs[2]]          # the seed still decides the tokens
    for i in range(6):
        engine.generate(prompts, max_tokens=2, temp=0.5 + 0.1 * i, top_k=8, top_p=0.9, seed=1, ignore_eos=True)
    assert engine.stats()["backends"] <= 4


def test_profile_lists_launchers_and_records_no_graph(models):
    from fastgguf_b200.engine.api import Engine
    d, cfg, W = models["b"]
    engine = Engine.from_dir(d, dtype="bfloat16", max_tokens=1024, max_batch=2)
    prompts = [[3, 5, 7, 11, 13], [2, 4]]
    plain = engine.generate(prompts, max_tokens=5, temp=0, ignore_eos=True, use_graphs=False)
    engine.profile(True)
    out = engine.generate(prompts, max_tokens=5, temp=0, ignore_eos=True)
    rows = engine.profile_report()
    engine.profile(False)
    assert [c.tokens for c in out] == [c.tokens for c in plain]              # eager steps: the same tokens
    names = {r["name"].split(" ")[0] for r in rows}
    assert rows and all(r["calls"] > 0 and r["ms"] > 0 for r in rows)
    assert "fg_gemm_tc" in names or "fg_gemm_generic" in names
    assert any(n.startswith("fg_attention") or n.startswith("fg_rope") for n in names)
    assert rows == sorted(rows, key=lambda r: -r["ms"])
    assert engine.profile_report() == []                                       # a report clears the records


def test_plain_kernels_switch_gives_the_same_tokens(models, monkeypatch):
    """FASTGGUF_PLAIN_KERNELS=1 puts a bfloat16 engine on the any-size kernels: the same results up to rounding."""
    from fastgguf_b200.engine.api import Engine
    from fastgguf_b200.engine.batch import StepEntry
    d, cfg, W = models["a"]
    toks = random_tokens(40, cfg["vocab_size"], 9)
    fast = Engine.from_dir(d, dtype="bfloat16", max_tokens=256, max_batch=1)
    monkeypatch.setenv("FASTGGUF_PLAIN_KERNELS", "1")
    slow = Engine.from_dir(d, dtype="bfloat16", max_tokens=256, max_batch=1)
    monkeypatch.delenv("FASTGGUF_PLAIN_KERNELS")
    got = []
    for e in (fast, slow):
        e.profile(True)
        s = e.acquire()
        got.append(np.asarray(e.step_host([StepEntry(s, toks, list(range(len(toks))))])))
        e.release(s)
        names = {r["name"].split(" ")[0] for r in e.profile_report()}
        e.profile(False)
        assert ("fg_gemm_tc" in names) == (e is fast) and ("fg_gemm_generic" in names) == (e is slow)
    want = plain_llama.plain_forward(cfg, W, toks).numpy()
    scale = np.abs(want).max()
    assert np.abs(got[1] - want).max() <= 1e-2 * scale and np.abs(got[0] - want).max() <= 1e-2 * scale


def test_float32_scratch_memory_is_shared_by_the_steps_of_an_engine():
    """Recorded float32 steps of 17 and more sequences and prompt steps use one block of scratch memory between them: a second width of the
    step, and a second sampler, add little, and what they compute stays the same while the block grows."""
    from helpers import TINY_B
    from fastgguf_b200.engine.api import Engine
    from fastgguf_b200.registry import config_from_dict
    cfg = dict(TINY_B, hidden_size=1024, num_attention_heads=16, num_key_value_heads=4, head_dim=64, intermediate_size=2048, vocab_size=32000)
    eng = Engine.from_random(config_from_dict(cfg), 3, dtype="float32", max_tokens=16384, max_batch=64)
    prompts = [[(7 * i + 3 * k) % 32000 for i in range(5 + k % 7)] for k in range(40)]

    def held(n, temp):
        """tokens, and how many MB of device memory came to be held"""
        before = torch.cuda.mem_get_info()[0]
        done = eng.generate(prompts[:n], temp=temp, top_k=4, max_tokens=5, seed=3, ignore_eos=True, use_graphs=True)
        torch.cuda.synchronize()
        return [c.tokens for c in done], (before - torch.cuda.mem_get_info()[0]) / 2 ** 20

    first = held(20, 0.0)                                  # planes of the head alone: 32,000 x 1,024 x 6 bytes, 188 MB
    assert first[1] > 150
    grown = [held(40, 0.0)[1], held(20, 0.5)[1], held(40, 0.5)[1]]
    assert max(grown) < 150, grown
    again = held(20, 0.0)
    assert again[0] == first[0]


def test_float32_steps_of_prompts_beside_running_sequences():
    """In a float32 step that brings a prompt and the next tokens of other sequences, the prompt's rows take the tiled attention kernel and the
    single tokens the any-size one, runs of them between prompts included; the logits are those of the sequences alone."""
    from helpers import TINY_B
    from fastgguf_b200 import StepEntry
    from fastgguf_b200.engine.api import Engine
    from fastgguf_b200.registry import config_from_dict
    cfg = dict(TINY_B, hidden_size=512, num_attention_heads=16, num_key_value_heads=4, head_dim=64, intermediate_size=1024, num_hidden_layers=2, max_position_embeddings=4096)
    eng = Engine.from_random(config_from_dict(cfg), 3, dtype="float32", max_tokens=16384, max_batch=8, max_seq_len=4096)
    rng = np.random.default_rng(5)
    draw = lambda n: [int(t) for t in rng.integers(0, cfg["vocab_size"], size=n)]  # noqa: E731
    running, prompts = [draw(1500), draw(70), draw(2900)], [draw(400), draw(333)]
    slots = [eng.acquire() for _ in running]
    eng.step_host([StepEntry(s, t[:-1], []) for s, t in zip(slots, running)])
    new = [eng.acquire() for _ in prompts]
    one = lambda i: StepEntry(slots[i], running[i][-1:], [0])  # noqa: E731
    whole = lambda i: StepEntry(new[i], prompts[i], [len(prompts[i]) - 1])  # noqa: E731
    eng.profile(True)
    got = eng.step_host([one(0), whole(0), one(1), one(2), whole(1)])
    calls = {r["name"].split(" ")[0]: r["calls"] for r in eng.profile_report()}
    eng.profile(False)
    layers = 2
    assert calls["fg_attention_prefill_f32"] == layers and calls["fg_attention_generic_kept"] == 2 * layers
    for logits, toks in zip(got, [running[0], prompts[0], running[1], running[2], prompts[1]]):
        s = eng.acquire()
        alone = eng.step_host([StepEntry(s, toks, [len(toks) - 1])])[0]
        eng.release(s)
        assert np.abs(logits - alone).max() <= 2e-5 * np.abs(alone).max()


def test_float32_steps_where_device_memory_is_short():
    """Without room for all of the scratch memory a float32 step takes its operands in more portions, with the same bits; without room for the
    least of it the plain chain computes the step."""
    import gc
    from helpers import TINY_B
    from fastgguf_b200 import StepEntry
    from fastgguf_b200.engine.api import Engine
    from fastgguf_b200.registry import config_from_dict
    cfg = dict(TINY_B, hidden_size=1024, num_attention_heads=16, num_key_value_heads=4, head_dim=64, intermediate_size=2048, vocab_size=32000)
    rng = np.random.default_rng(5)
    toks = [int(t) for t in rng.integers(0, 32000, size=40)]

    def logits(left):
        """of every place of a prompt, in an engine that has `left` bytes of device memory left (None: all of it); the head's planes are 188 MB"""
        eng = Engine.from_random(config_from_dict(cfg), 3, dtype="float32", max_tokens=1024, max_batch=2)
        s = eng.acquire()
        eng.step_host([StepEntry(s, toks[:8], [7])])       # (activations, modules; eight rows need no scratch memory)
        eng.release(s)
        hold = None
        if left is not None:
            torch.cuda.synchronize()
            hold = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
        try:
            eng.profile(True)
            s = eng.acquire()
            got = np.array(eng.step_host([StepEntry(s, toks, list(range(40)))]))
            names = {r["name"] for r in eng.profile_report()}
            eng.profile(False)
        finally:
            del hold
            torch.cuda.empty_cache()
        del eng
        gc.collect()
        return got, any(n.startswith("fg_gemm_f32_tc") for n in names)

    gib = 1 << 30
    want, planes = logits(None)
    assert planes
    portions, planes = logits(gib + (120 << 20))
    assert planes and np.array_equal(portions, want)
    plain, planes = logits(gib - (100 << 20))
    assert not planes and 0 < np.abs(plain - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_busy_default_stream_changes_nothing(models, dtype):
    """The engine's stream does not wait for the default stream.  Whatever an engine, a sampler and a recorded step set up before their first
    use is therefore queued on the engine's own stream: a thread that keeps the default stream milliseconds behind must not delay it."""
    import threading
    from fastgguf_b200.engine.api import Engine
    d, cfg, _ = models["b"]
    prompts = [random_tokens(n, cfg["vocab_size"], 70 + i) for i, n in enumerate([9, 30, 2])]

    def outputs():
        engine = Engine.from_dir(d, dtype=dtype, max_tokens=1024, max_batch=4)
        return [[c.tokens for c in engine.generate(prompts, temp=t, top_k=20, top_p=0.9, repeat_penalty=1.2, seed=3, max_tokens=12, ignore_eos=True)]
                for t in (0, 0.7)]

    want, stop, idle = outputs(), threading.Event(), torch.cuda.Event()

    def keep_busy():
        while not stop.is_set():
            for _ in range(8):
                torch.cuda._sleep(2_000_000)                  # about a millisecond each
            idle.record()
            idle.synchronize()

    t = threading.Thread(target=keep_busy)
    t.start()
    try:
        got = [outputs() for _ in range(3)]
    finally:
        stop.set()
        t.join()
    assert all(g == want for g in got)


def test_a_session_step_that_is_refused_queues_nothing(models):
    """A step that names a sequence which has left its batch is refused before page-table entries are on their way to the device, and the
    steps behind it find what they would have found without it."""
    from fastgguf_b200.engine.api import Engine
    from fastgguf_b200.engine.batch import StepEntry
    from fastgguf_b200 import SamplingParams
    d, cfg, _ = models["b"]
    prompts = [random_tokens(n, cfg["vocab_size"], 80 + i) for i, n in enumerate([61, 5, 62])]

    def run(with_refused_calls):
        engine = Engine.from_dir(d, dtype="float32", max_tokens=2048, max_batch=4)
        session = engine.session(prompts, SamplingParams(temp=0.0))
        session.advance([0, 1, 2])
        for step in range(70):                               # sequences 0 and 2 come to new pages one step after the other
            session.advance([0, 2])
            if with_refused_calls:
                before = engine.stats()
                with pytest.raises(Exception, match="left this batch"):
                    session.advance([0, 2, 1])
                assert engine.stats() == before
        slots = [session.slots[0], session.slots[2]]
        return engine.step_host([StepEntry(s, [7, 8], [0, 1]) for s in slots])

    assert np.array_equal(run(True), run(False))


@pytest.mark.parametrize("heads,kv_heads,lengths,tiles", [(8, 8, [17], False), (8, 8, [33], False), (8, 8, [33] * 4, True), (8, 8, [200], True),
                                                          (4, 1, [64], False), (4, 1, [17] * 4, False), (32, 8, [17], False), (32, 8, [17] * 4, True)])
def test_float32_prompts_take_the_kernel_that_is_done_first(heads, kv_heads, lengths, tiles):
    """A few new tokens are the any-size kernel's, unless there are so many such sequences that their tiles, side by side, are done first."""
    from helpers import TINY_B
    from fastgguf_b200.engine.api import Engine
    from fastgguf_b200.registry import config_from_dict
    cfg = dict(TINY_B, hidden_size=512, num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=64, intermediate_size=512, vocab_size=256)
    engine = Engine.from_random(config_from_dict(cfg), 3, dtype="float32", max_tokens=2048, max_batch=4)
    engine.profile(True)
    engine.generate([random_tokens(n, 256, 90 + i) for i, n in enumerate(lengths)], temp=0, max_tokens=1, ignore_eos=True)
    names = {r["name"].split(" ")[0] for r in engine.profile_report()}
    engine.profile(False)
    assert ("fg_attention_prefill_f32" in names) == tiles and any(n.startswith("fg_attention_generic") for n in names) == (not tiles), names
