"""Prompt steps of 16 to 64 rows: the tensor-memory attention kernel already runs in them, beside contractions that count them as small."""
import os
import re

import numpy as np
import pytest


def test_kernels_beside_attention_do_not_go_by_the_number_of_rows():
    """A kernel that stands between the tensor-memory attention kernel and a contraction, and released its successor at its start, would
    let the contraction start beside attention.  Whether it may is the host's to say (`early`): the step's rows do not tell."""
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fastgguf_b200", "csrc")
    for name, kernels in (("attention_prep.cu", ("qkv_prepare_kernel", "differential_combine_kernel", "head_gate_kernel")),
                          ("attention_latent.cu", ("gate_slice_kernel", "latent_expand_kernel")), ("elementwise.cu", ("rmsnorm_pair_kernel",)),
                          ("gemm_generic.cu", ("gemm_generic_kernel", "gemv_rows_kernel", "gemv_splitk_kernel"))):
        with open(os.path.join(csrc, name)) as f:
            text = f.read()
        for k in kernels:
            body = text[text.index(k + "("):]
            body = body[:body.index("pdl_wait();")]
            assert "small_step" not in body, k
            assert re.sub(r"if \(early\) pdl_launch_dependents\(\);", "", body).count("pdl_launch_dependents") == 0, k


def test_recurrences_release_the_output_projection_early_in_small_steps_alone():
    """The last kernel of a recurrence stands between two contractions.  In a step of more than 64 rows both hold tensor memory, and one that
    released its successor at its start would let the second start beside the first.  How many rows a step has is not its number of
    sequences, which is the grid of the token-by-token kernels."""
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fastgguf_b200", "csrc")
    for name, by_rows, at_the_end in (("retention.cu", ("retention_seq_kernel", "retention_regs_kernel"), ("retention_chunk_out_kernel", "retention_chunk_out_fast")),
                                      ("gla.cu", ("gla_seq_kernel",), ("gla_chunk_out_kernel",))):
        with open(os.path.join(csrc, name)) as f:
            text = f.read()
        for k in by_rows + at_the_end:
            body = text[text.index(k + "(const"):]
            body = body[:body.index("row0 = " if k in by_rows else "const int c =")]
            assert re.findall(r"pdl_launch_dependents\w*\([^;]*;", body) == ["pdl_launch_dependents_small_step(cu_rows[gridDim.x]);"] * (k in by_rows), k


def test_the_norm_between_contractions_goes_by_the_rows_of_the_step():
    """A final norm has as many blocks as rows are wanted, behind a contraction of all the step's rows: the host says whether it may release the
    head's contraction at its start."""
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fastgguf_b200", "csrc")
    with open(os.path.join(csrc, "elementwise.cu")) as f:
        text = f.read()
    for k in ("void rmsnorm_kernel(", "rmsnorm_regs_kernel("):
        body = text[text.index(k):]
        assert re.findall(r".*pdl_launch_dependents.*", body[:body.index("pdl_wait();")]) == ["    if (early) pdl_launch_dependents();"], k
    with open(os.path.join(csrc, "host", "parts.cpp")) as f:
        text = f.read()
    calls = [line for line in text.splitlines() if "fg_rmsnorm," in line and "FG_LAUNCH" in line]
    assert calls and all("FG_LAUNCH_STEP" in line and "rt.early_between(x.rows)" in line for line in calls)


def _saluzen():
    from saluzen_cases import attn, config, delta, dense, latent, parallel, parallel_2, ssm
    left = dict(heads=16, kv_heads=4, dim=64, vdim=64, scale=0.125)
    return config(1024, 4096, [
        (latent(16, 64, 64, 64, 256, 768, 0.09, 10000.0), dense(4096)),
        (latent(16, 64, 64, 64, 256, 768, 0.09, 10000.0, kv_from=0), dense(4096)),
        (parallel(attn(**left, rot=(500000.0, 32), scaling=(8.0, 1.0, 4.0, 8192)), ssm(16, 64, 128, 1, 4, 1)), dense(4096)),
        (parallel_2(attn(**left, rot=(1000000.0, 32), size=512), delta(8, 4, 128, 128, 4), 0.9, 0.4), dense(4096))], eps=1e-6)


def _pirozen():
    from pirozen_cases import attention, config, moe
    att = attention(16, 4, 64, 64, 0.125, size=512, rot=(1000000.0, 32), scaling=(8.0, 4096, 32.0, 1.0))
    return config(1024, 4096, [(att, moe(1024, 6, 2, scale=2.0, identity=2, groups=(2, 1), shared=1024))] * 4, loop=(0, 4, 1), side=128, eps=1e-6)


def _buguzen():
    from buguzen_cases import config, differential, keys_as_values, lightning
    return config(1024, 4096, [
        (differential(8, 4, 64, 128, 0.125, 0.5, size=512, rot=(10000.0, 32), scaling=(2.0,)), 4096),
        (keys_as_values(8, 2, 128, 0.09, size=700, rot=(200000.0, 64), scaling=(16.0, 1.0, 3.0, 2048)), 4096),
        (lightning(8, 128, 128, [0.5, 0.8, 0.9, 0.95, 0.98, 0.99, 0.995, 0.999]), 4096)], loop=(0, 3, 2), side=256)


@pytest.mark.gpu
@pytest.mark.parametrize("case", [_saluzen, _pirozen, _buguzen])
def test_many_short_prompt_steps_back_to_back(case):
    """Two hundred prompt steps of one to three sequences, 16 to 64 rows in all, one after another, every tenth followed by a decode step:
    each ends with finite logits, and a repeated prompt gives the same."""
    from fastgguf_b200.engine.api import Engine
    from fastgguf_b200.engine.batch import StepEntry
    from fastgguf_b200.registry import config_from_dict
    eng = Engine.from_random(config_from_dict(case()), 3, dtype="bfloat16", max_tokens=4096, max_batch=4, max_seq_len=1024)
    rng = np.random.default_rng(5)
    draw = lambda n: [int(t) for t in rng.integers(0, 4096, size=n)]  # noqa: E731
    fixed, first = [draw(n) for n in (16, 17, 31)], None
    for i in range(200):
        total = int(rng.integers(16, 65))
        cut = sorted(rng.choice(np.arange(1, total), size=int(rng.integers(0, 3)), replace=False).tolist())
        toks = fixed if i % 4 == 0 else [draw(b - a) for a, b in zip([0] + cut, cut + [total])]
        slots = [eng.acquire() for _ in toks]
        got = eng.step_host([StepEntry(s, t, [len(t) - 1]) for s, t in zip(slots, toks)])
        assert np.isfinite(got).all()
        if i % 4 == 0:
            first = got if first is None else first
            assert np.array_equal(got, first)
        if i % 10 == 0:
            assert np.isfinite(eng.step_host([StepEntry(s, draw(1), [0]) for s in slots])).all()
        for s in slots:
            eng.release(s)
    eng.cache.check()


def _zirivik():
    from zirivik_cases import config, dense, retention
    decay = [1.0 - 2.0 ** (-5 - h / 2) for h in range(8)]
    return config(1024, 4096, [(retention(8, 128, 128, decay, (10000.0, 64)), dense(4096)), (retention(8, 64, 64, decay), dense(4096))] * 2)


def _salulorn():
    from salulorn_cases import config, dense, gla
    return config(512, 2048, [(gla(8, 64, 64, 16.0, 16), dense(1024))] * 4)


@pytest.mark.gpu
@pytest.mark.parametrize("case", [_zirivik, _salulorn])
def test_many_steps_of_many_short_portions(case, tmp_path):
    """One hundred and fifty steps of 8 to 80 sequences with 2 to 15 tokens each, more than 64 rows in all, which the token-by-token kernels
    walk between two tensor-memory contractions, every tenth followed by a step of one token for each: all end with finite logits."""
    from fastgguf_b200.engine.api import Engine
    from fastgguf_b200.engine.batch import StepEntry
    from fastgguf_b200.registry import config_from_dict
    room = dict(dtype="bfloat16", max_tokens=16384, max_batch=80, max_seq_len=256)
    if case is _salulorn:                                    # (the rank of a decay is a shape of its weights)
        import salulorn_cases
        eng = Engine.from_dir(salulorn_cases.make_model(tmp_path, case(), 3)[0], **room)
    else:
        eng = Engine.from_random(config_from_dict(case()), 3, **room)
    rng = np.random.default_rng(6)
    draw = lambda n: [int(t) for t in rng.integers(0, 2048, size=n)]  # noqa: E731
    for i in range(150):
        lengths = rng.integers(2, 16, size=int(rng.integers(8, 81)))
        lengths[0] += max(0, 65 - int(lengths.sum())) if i % 2 else 0
        toks = [draw(int(n)) for n in lengths]
        slots = [eng.acquire() for _ in toks]
        assert np.isfinite(eng.step_host([StepEntry(s, t, [len(t) - 1]) for s, t in zip(slots, toks)])).all()
        if i % 10 == 0:
            assert np.isfinite(eng.step_host([StepEntry(s, draw(1), [0]) for s in slots])).all()
        for s in slots:
            eng.release(s)
    eng.cache.check()
