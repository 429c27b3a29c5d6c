"""Steps of 17 to 129 rows at the serving models' widths: prompts on both sides of the stream form's limit, and the captured decode steps of
the 32-bit path that run on the split product."""
import pytest
import torch

import plain_lfm2

pytestmark = pytest.mark.gpu


def _model(tmp_path, sizes, seed, dtype):
    from conftest import serving_width_config
    from vapi_b200.weights import write_random_model
    cfg = serving_width_config(sizes)
    d = write_random_model(str(tmp_path / "m"), cfg, seed, std=0.02, norm_init="perturbed", dtype=dtype)
    return d, plain_lfm2.PlainLfm2(d), cfg


def _tokens(n, seed, vocab):
    return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def test_prompts_on_both_sides_of_the_stream_forms_limits(tmp_path):
    """One prompt of 32 to 129 tokens, and a portion beside decoding requests with as many rows in all: the blocks run in their stream form up
    to 128 rows (tiles of 64 and of 128 tokens), and the logits are the plain model's within bfloat16 rounding."""
    from vapi_b200 import ops
    from vapi_b200.engine.runner import ModelRunner
    from vapi_b200.engine.step import StepEntry
    d, plain, cfg = _model(tmp_path, "700m", 5, torch.bfloat16)
    r = ModelRunner.from_dir(d, dtype="bfloat16", num_pages=80, max_requests=24, max_batched_tokens=1024, max_context=256)
    seen, real = [], r._forward_few_rows
    r._forward_few_rows = lambda ctx, views: (seen.append(ctx.n), real(ctx, views))[1]

    def check(logits, toks):
        want = plain.logits(toks)[-1]
        span = float(want.max() - want.min())
        assert float((logits.float().cpu() - want).abs().max()) < 0.02 * span

    opened = 0
    for n in (32, 33, 64, 65, 100, 127, 128, 129):
        toks = _tokens(n, n, cfg["vocab_size"])
        rc = r.cache.open(opened)
        opened += 1
        assert r.cache.reserve(rc, n)
        check(r.step([StepEntry(rc, toks, [n - 1])])[0], toks)
        r.cache.close(rc)
    assert seen == [n for n in (32, 33, 64, 65, 100, 127, 128, 129) if n <= ops.STREAM_PROMPT_MAX_ROWS] and ops.STREAM_PROMPT_MAX_ROWS == 128
    # nine requests decode beside a portion
    del seen[:]
    prompts = [_tokens(5 + 3 * i, 90 + i, cfg["vocab_size"]) for i in range(9)]
    rcs = [r.cache.open(100 + i) for i in range(9)]
    for rc, p in zip(rcs, prompts):
        assert r.cache.reserve(rc, len(p) + 4)
    r.step([StepEntry(rc, p, []) for rc, p in zip(rcs, prompts)])
    del seen[:]
    for at, n in enumerate((24, 56, 119, 120)):
        toks = _tokens(n, 50 + n, cfg["vocab_size"])
        rc = r.cache.open(opened)
        opened += 1
        assert r.cache.reserve(rc, n)
        entries = [StepEntry(q, [200 + at], [0]) for q in rcs] + [StepEntry(rc, toks, [n - 1])]
        logits = r.step(entries)
        check(logits[9], toks)
        check(logits[4], prompts[4] + [200 + i for i in range(at + 1)])
        r.cache.close(rc)
    assert seen == [33, 65, 128]
    r.check_status()


def test_captured_float32_decode_on_the_split_product(tmp_path):
    """24 requests in float32: the bucket of 32 rows, whose wide products split floats for the tensor cores (scratch from the graph's memory,
    clusters and dependent launches in the capture).  Captured against eager, and against the plain model."""
    from vapi_b200 import ops
    from vapi_b200.engine.runner import ModelRunner
    from vapi_b200.engine.step import StepEntry
    d, plain, cfg = _model(tmp_path, "700m", 6, torch.float32)
    assert ops.linear_f32_pays(32, 3 * cfg["hidden_size"], cfg["hidden_size"])
    prompts = [_tokens(3 + (7 * i) % 40, 300 + i, cfg["vocab_size"]) for i in range(24)]
    rows = {}
    for graphs in (True, False):
        r = ModelRunner.from_dir(d, dtype="float32", num_pages=60, max_requests=32, max_batched_tokens=1024, max_context=256)
        rcs = [r.cache.open(i) for i in range(24)]
        for rc, p in zip(rcs, prompts):
            assert r.cache.reserve(rc, len(p) + 3)
        r.step([StepEntry(rc, p, []) for rc, p in zip(rcs, prompts)])
        for s in range(3):                                 # (the graph is replayed twice behind the step that captured it)
            entries = [StepEntry(rc, [100 + i + s], [0]) for i, rc in enumerate(rcs)]
            lg = r.step_decode_graph(entries) if graphs else r.step(entries)
            assert lg is not None
        rows[graphs] = lg.cpu().clone()
        r.check_status()
        if graphs:
            assert r._graphs[32] is not None
    want = torch.stack([plain.logits(p + [100 + i + s for s in range(3)])[-1] for i, p in enumerate(prompts)])
    span = float(want.max() - want.min())
    # (bound: three layers and the head of float32 sums of at most 6,912 terms, some 1e-6 of what they add up)
    assert float((rows[True] - want).abs().max()) < 3e-5 * span and float((rows[False] - want).abs().max()) < 3e-5 * span


@pytest.mark.parametrize("S", [33, 47, 64])
def test_decode_steps_of_33_to_64_requests_in_the_stream_form(tmp_path, S):
    """The bucket of 64 rows, captured, and the step as it is, eager (33 and 47 rows of a tile of 64 tokens): both run the blocks' stream
    form, and the logits are the plain model's within bfloat16 rounding."""
    from vapi_b200.engine.runner import ModelRunner
    from vapi_b200.engine.step import StepEntry
    d, plain, cfg = _model(tmp_path, "700m", 7, torch.bfloat16)
    prompts = [_tokens(3 + (5 * i) % 23, 400 + i, cfg["vocab_size"]) for i in range(S)]
    for graphs in (True, False):
        r = ModelRunner.from_dir(d, dtype="bfloat16", num_pages=160, max_requests=64, max_batched_tokens=1024, max_context=128)
        r._graphs_off = not graphs
        seen, real = [], r._forward_few_rows
        r._forward_few_rows = lambda ctx, views: (seen.append((ctx.n, ctx.max_q)), real(ctx, views))[1]
        rcs = [r.cache.open(i) for i in range(S)]
        for rc, p in zip(rcs, prompts):
            assert r.cache.reserve(rc, len(p) + 2)
        for i in range(0, S, 16):
            r.step([StepEntry(rc, p, []) for rc, p in zip(rcs[i:i + 16], prompts[i:i + 16])])
        del seen[:]
        for at in range(2):
            entries = [StepEntry(rc, [200 + at], [0]) for rc in rcs]
            logits = r.step_decode_graph(entries) if graphs else r.step(entries)
        assert seen and set(seen) == {(64 if graphs else S, 1)}
        for i in (0, S // 2, S - 1):
            want = plain.logits(prompts[i] + [200, 201])[-1]
            assert float((logits[i].float().cpu() - want).abs().max()) < 0.02 * float(want.max() - want.min())
        r.check_status()
