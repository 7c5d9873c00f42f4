"""The engine's step function on the GPU against the plain implementation: every way of
cutting the same requests into steps must give the same logits, in 32-bit and bfloat16."""

from __future__ import annotations

import itertools

import pytest
import torch

from harness import (PAGE_TOKENS, TOLERANCE, assert_close, gpu_runner, make_tensors, plain_logits,
                     tiny_config, tokens_for)
from mini_gpt_inference_b200.engine.runner import StepEntry

pytestmark = pytest.mark.gpu

CASES = (list(itertools.product("AB", ["float32", "bfloat16"], [False, True]))
         + [("C", "float32", False), ("C", "bfloat16", False)])
IDS = [f"{w}-{d}-{'sharp' if s else 'soft'}" for w, d, s in CASES]


def _setup(which, dtype, sharp, num_pages=64, seed=3):
    cfg = tiny_config(which)
    tensors = make_tensors(cfg, seed, dtype, sharp)
    runner = gpu_runner(cfg, tensors, dtype, PAGE_TOKENS[which], num_pages)
    # A sharpened softmax amplifies bfloat16 rounding of q and k; 32-bit is unaffected.
    tol = TOLERANCE[dtype] * (4 if sharp and dtype == "bfloat16" else 1)
    return cfg, tensors, runner, tol


@pytest.mark.parametrize("which,dtype,sharp", CASES, ids=IDS)
def test_whole_prompt_alone(which, dtype, sharp):
    cfg, tensors, runner, tol = _setup(which, dtype, sharp)
    for length, seed in [(cfg.n_positions, 1), (37, 2), (1, 3), (2, 4), (PAGE_TOKENS[which] + 1, 5)]:
        tokens = tokens_for(cfg, length, seed)
        want = plain_logits(cfg, tensors, tokens)
        got = runner.step([StepEntry("r", tokens, list(range(length)))])
        runner.finish("r")
        assert got.shape == (length, cfg.vocab_size) and got.dtype == torch.float32
        assert_close(got, want, tol, f"whole prompt of {length}")
    runner.manager.check()
    assert runner.manager.stats()["allocated_blocks"] == 0


@pytest.mark.parametrize("which,dtype,sharp", CASES, ids=IDS)
def test_last_32_tokens_one_by_one(which, dtype, sharp):
    cfg, tensors, runner, tol = _setup(which, dtype, sharp)
    length = cfg.n_positions
    tokens = tokens_for(cfg, length, 7)
    want = plain_logits(cfg, tensors, tokens)
    head = length - 32
    outs = [runner.step([StepEntry("r", tokens[:head], list(range(head)))])]
    for t in range(head, length):
        outs.append(runner.step([StepEntry("r", tokens[t: t + 1], [0])]))
    assert_close(torch.cat(outs), want, tol, "prefill then 32 single tokens")


@pytest.mark.parametrize("which,dtype,sharp", CASES, ids=IDS)
def test_portions_of_changing_size(which, dtype, sharp):
    cfg, tensors, runner, tol = _setup(which, dtype, sharp)
    length = cfg.n_positions - 3
    tokens = tokens_for(cfg, length, 8)
    want = plain_logits(cfg, tensors, tokens)
    sizes = itertools.cycle([13, 7, 2, 5, 2, 1, 3, 16, 2, 9])
    outs, pos = [], 0
    while pos < length:
        n = min(next(sizes), length - pos)
        outs.append(runner.step([StepEntry("r", tokens[pos: pos + n], list(range(n)))]))
        pos += n
    assert_close(torch.cat(outs), want, tol, "portions of changing size")


@pytest.mark.parametrize("which,dtype,sharp", CASES, ids=IDS)
def test_mixed_requests_with_page_reuse(which, dtype, sharp):
    """Up to four live requests; portions of some beside decoded tokens of others; a pool so
    small that the pages of finished requests are handed out again."""
    cfg = tiny_config(which)
    pt = PAGE_TOKENS[which]
    lengths = [cfg.n_positions, 29, cfg.n_positions - 9, 3, 41, 2 * pt, 17, cfg.n_positions // 2]
    # room for the four longest at once, no more
    pool = sum(sorted(-(-n // pt) for n in lengths)[-4:])
    cfg, tensors, runner, tol = _setup(which, dtype, sharp, num_pages=pool)
    # Every cache row starts as NaN and a finished request's pages become NaN again: a query that
    # reads a row its own request did not write (beyond its length, or left by the page's last
    # holder) turns its logits into NaN.
    for pages in runner.storage.k + runner.storage.v:
        pages.fill_(float("nan"))
    reqs = {f"q{i}": tokens_for(cfg, n, 20 + i) for i, n in enumerate(lengths)}
    want = {rid: plain_logits(cfg, tensors, toks) for rid, toks in reqs.items()}
    got = {rid: [] for rid in reqs}
    waiting = list(reqs)
    live: dict[str, int] = {}
    sizes = itertools.cycle([5, 1, 2, 11, 1, 1, 7, 3, 1, 2])
    gen = torch.Generator().manual_seed(99)
    steps = 0
    while waiting or live:
        while waiting and len(live) < 4:
            live[waiting.pop(0)] = 0
        entries, order = [], []
        for rid in list(live):
            if len(live) > 1 and torch.rand((), generator=gen).item() < 0.25:
                continue                                   # left out of this step
            pos = live[rid]
            n = min(next(sizes), len(reqs[rid]) - pos)
            entries.append(StepEntry(rid, reqs[rid][pos: pos + n], list(range(n))))
            order.append((rid, n))
            live[rid] = pos + n
        if not entries:
            continue
        logits = runner.step(entries)
        row = 0
        for rid, n in order:
            got[rid].append(logits[row: row + n])
            row += n
        for rid in [r for r, p in live.items() if p == len(reqs[r])]:
            held = torch.tensor([p for p in runner.manager.block_table(rid, 0) if p >= 0],
                                dtype=torch.long, device="cuda")
            runner.finish(rid)
            for pages in runner.storage.k + runner.storage.v:
                pages[:, held] = float("nan")
            del live[rid]
        runner.manager.check()
        steps += 1
    assert runner.manager.stats()["allocated_blocks"] == 0
    for rid in reqs:
        assert not torch.isnan(torch.cat(got[rid])).any(), f"request {rid} read a cache row that was not its own"
        assert_close(torch.cat(got[rid]), want[rid], tol, f"mixed batch, request {rid}")


@pytest.mark.parametrize("which,dtype", [("A", "float32"), ("B", "bfloat16"), ("A", "bfloat16")])
def test_prompt_steps_of_a_repeated_shape_are_replayed(which, dtype):
    """A step shape that comes a second time is captured and replayed from then on (different
    tokens, other pages, a request beside it): the logits stay those of the plain
    implementation, and equal those of a runner that never captures."""
    cfg, tensors, runner, tol = _setup(which, dtype, False)
    _, _, eager, _ = _setup(which, dtype, False)
    eager.use_cuda_graphs = False
    n = min(23, cfg.n_positions - 6)
    outs = []
    for rep in range(5):
        a, b = tokens_for(cfg, n + 5, 40 + rep), tokens_for(cfg, 6, 60 + rep)
        want_a, want_b = plain_logits(cfg, tensors, a), plain_logits(cfg, tensors, b)
        for r in (runner, eager):
            r.step([StepEntry("a", a[:5], [])])                      # another shape in between
            got = r.step([StepEntry("a", a[5:], list(range(n))), StepEntry("b", b, [5, 0])])
            assert_close(got[:n], want_a[5:], tol, f"repeat {rep}, request a")
            assert_close(got[n:], want_b[[5, 0]], tol, f"repeat {rep}, request b")
            outs.append(got)
            r.finish("a")
            if rep % 2 == 0:
                r.finish("b")                                      # b's pages change every other time
            else:
                r.step([StepEntry("b", [1], [])])
                r.finish("b")
    assert runner.shape_graph_replays >= 3 and eager.shape_graph_replays == 0
    for mine, theirs in zip(outs[0::2], outs[1::2]):
        if dtype == "float32":
            assert torch.equal(mine, theirs), "a replayed step differs from the same launches run eagerly"
        else:
            # The fused feed-forward of small steps adds its CTAs' partial sums in whatever order
            # they arrive, so a 32-bit sum can differ in its last bit between a replayed and an
            # eagerly launched kernel; once in twenty steps such a bit moves an activation or a
            # cached key to the neighbouring bfloat16 value (measured: up to 1.4e-3 on these
            # logits).  Equal up to a few such roundings, far inside the bound against the plain
            # logits, is what the same launches guarantee in bfloat16; bit for bit only in 32-bit.
            diff = float((mine - theirs).abs().max())
            assert diff <= tol / 2, f"a replayed step differs from the same launches run eagerly by {diff:.3e}"
    runner.manager.check()


@pytest.mark.parametrize("which,dtype", list(itertools.product("AB", ["float32", "bfloat16"])))
def test_head_behind_a_replayed_step(which, dtype):
    """Logits too large to be copied out of a graph are computed behind it: the plain ones, in a tensor that later steps
    leave alone."""
    cfg, tensors, runner, tol = _setup(which, dtype, False)
    runner.HEAD_APART_BYTES, runner.HEAD_APART_ROWS = 0, 2
    n = cfg.n_positions - 1
    outs = []
    for rep in range(5):
        tokens = tokens_for(cfg, n, 90 + rep)
        outs.append((tokens, runner.step([StepEntry("r", tokens, list(range(n)))])))
        runner.finish("r")
    assert runner.shape_graph_replays == 3
    for tokens, got in outs:
        assert_close(got, plain_logits(cfg, tensors, tokens), tol, "the head behind a replayed step")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_no_matrix_is_said_to_follow_the_head_of_a_replayed_step(dtype):
    """A head behind a replayed step follows nothing that the kernel set saw: a hint from whatever ran last, the head of the replay
    before it or another model's matrix, would have later steps ask the wrong matrix into L2."""
    cfg, tensors, runner, tol = _setup("A", dtype, False)
    other = _setup("B", dtype, False)
    runner.HEAD_APART_BYTES, runner.HEAD_APART_ROWS = 0, 2
    ops, head, n = runner.ops, runner.model.head.embedding.weight, cfg.n_positions - 1
    assert other[2].ops is ops                                            # (models of a device share it)
    for rep in range(4):
        if rep == 3:
            other[2].step([StepEntry("o", tokens_for(other[0], 9, 1), [8])])      # another model's pass in between
            last = ops._last_weight
        ops._next_weight.clear()
        tokens = tokens_for(cfg, n, 90 + rep)
        got = runner.step([StepEntry("r", tokens, list(range(n)))])
        if rep >= 2:
            assert head.data_ptr() not in ops._next_weight and not ops._next_weight        # a replay and its head: no hint at all
        if rep < 3:
            runner.finish("r")
    assert runner.shape_graph_replays == 2 and last is not None
    # and a decode step behind it is right
    more = runner.step([StepEntry("r", [5], [0])])
    want = plain_logits(cfg, tensors, tokens + [5])
    assert_close(torch.cat([got, more]), want, tol, "a decode step behind a replayed step's head")


@pytest.mark.parametrize("family,which", [("fakilorn", "A"), ("nogatar", "A"), ("nogatar", "B")])
def test_other_heads_behind_a_replayed_step(family, which):
    """Heads with a scale and heads of their own matrix with a cap, behind replayed steps and with decode steps after them."""
    import importlib

    from mini_gpt_inference_b200 import FakilornConfig, NogatarConfig
    from mini_gpt_inference_b200.engine.build import load_model, make_runner
    from mini_gpt_inference_b200.kernels.ops import default_ops

    cases = importlib.import_module(f"{family}_cases")
    raw = cases.config(which)
    tensors = cases.random_weights(raw, 5)
    kind = {"fakilorn": FakilornConfig, "nogatar": NogatarConfig}[family]
    loaded = load_model(config=kind.from_dict(raw), tensors=tensors, dtype="float32", device="cuda:0")
    runner = make_runner(loaded, default_ops("cuda:0"), 8, 40, 2)
    runner.HEAD_APART_BYTES, runner.HEAD_APART_ROWS = 0, 2
    n = 67
    for rep in range(4):
        tokens = cases.tokens_for(raw, n + 2, 60 + rep)
        got = [runner.step([StepEntry("r", tokens[:n], list(range(n)))])]
        got += [runner.step([StepEntry("r", tokens[t: t + 1], [0])]) for t in (n, n + 1)]
        runner.finish("r")
        cases.assert_rows_close(torch.cat(got), cases.plain_logits(raw, tensors, tokens), 3e-4, f"{family} {which}, pass {rep}")
    assert runner.shape_graph_replays == 2


def test_captured_shapes_are_bounded():
    cfg, tensors, runner, tol = _setup("A", "bfloat16", False)
    runner.SHAPE_GRAPHS = 3
    for n in (2, 3, 4, 5, 6, 7):
        for rep in range(3):
            tokens = tokens_for(cfg, n, 80 + n)
            got = runner.step([StepEntry("r", tokens, [n - 1])])
            assert_close(got, plain_logits(cfg, tensors, tokens)[-1:], tol, f"{n} tokens, repeat {rep}")
            runner.finish("r")
    assert len(runner._shape_graphs) == 3 and runner.shape_graph_replays == 6


@pytest.mark.parametrize("which,dtype", [("A", "float32"), ("B", "float32")])
def test_cuttings_agree_bitwise_in_32bit(which, dtype):
    """In 32-bit every (token, head) and every output element is computed by the same
    instruction sequence however the batch is cut, so the logits are equal bit for bit."""
    cfg, tensors, runner, _ = _setup(which, dtype, False)
    tokens = tokens_for(cfg, 50, 11)
    whole = runner.step([StepEntry("a", tokens, list(range(50)))])
    other = tokens_for(cfg, 23, 12)
    runner.step([StepEntry("o", other[:9], [])])
    outs = [runner.step([StepEntry("b", tokens[:20], list(range(20))), StepEntry("o", other[9:10], [0])])[:20]]
    outs.append(runner.step([StepEntry("o", other[10:23], []), StepEntry("b", tokens[20:50], list(range(30)))]))
    assert torch.equal(torch.cat(outs), whole)


def test_step_errors_are_clear():
    cfg, tensors, runner, _ = _setup("A", "float32", False, num_pages=4)
    from mini_gpt_inference_b200.cache import CacheFullError
    from mini_gpt_inference_b200.engine.runner import StepError

    with pytest.raises(StepError, match="vocabulary"):
        runner.step([StepEntry("x", [cfg.vocab_size], [0])])
    with pytest.raises(StepError, match="position table"):
        runner.step([StepEntry("x", [1] * (cfg.n_positions + 1), [])])
    with pytest.raises(StepError, match="wants logits"):
        runner.step([StepEntry("x", [1, 2], [2])])
    runner.step([StepEntry("x", [1] * 60, [])])
    with pytest.raises(CacheFullError):
        runner.step([StepEntry("y", [1] * 20, [])])
    runner.manager.check()


@pytest.mark.parametrize("which,dtype", list(itertools.product("ABC", ["float32", "bfloat16"])))
def test_released_request_is_recomputed_to_the_same_logits(which, dtype):
    """Preemption by recomputation, seen from the step function: a request that has run through its
    prompt and a few single tokens gives everything back, other requests take its pages, and it
    comes again from position 0 with prompt and generated tokens as one prompt in portions of 13
    beside the others' decoding.  Its logits, first pass and second, are the plain ones at every
    position (the reference checks tokens only, tests/test_paged.py:107-143)."""
    cfg = tiny_config(which)
    pt = PAGE_TOKENS[which]
    n = cfg.n_positions
    cfg, tensors, runner, tol = _setup(which, dtype, False, num_pages=2 * (-(-n // pt)) + 2)
    victim, other, late = tokens_for(cfg, n - 5, 31), tokens_for(cfg, n // 2, 32), tokens_for(cfg, n // 3, 33)
    want = {k: plain_logits(cfg, tensors, v) for k, v in (("v", victim), ("o", other), ("l", late))}
    for pages in runner.storage.k + runner.storage.v:
        pages.fill_(float("nan"))
    # first pass: most of the prompt, then single tokens beside another request
    first = n // 2
    got = [runner.step([StepEntry("v", victim[:first], list(range(first))), StepEntry("o", other[:7], [])])[:first]]
    pos_o = 7
    for t in range(first, first + 6):
        out = runner.step([StepEntry("v", victim[t: t + 1], [0]), StepEntry("o", other[pos_o: pos_o + 1], [0])])
        got.append(out[:1])
        assert_close(out[1:], want["o"][pos_o: pos_o + 1], tol, "the other request, first pass")
        pos_o += 1
    assert_close(torch.cat(got), want["v"][: first + 6], tol, "first pass of the request")
    # it gives way; a newcomer takes pages (some of them the ones just freed)
    held = [p for p in runner.manager.block_table("v", 0) if p >= 0]
    runner.finish("v")
    for pages in runner.storage.k + runner.storage.v:
        pages[:, torch.tensor(held, device="cuda")] = float("nan")
    out = runner.step([StepEntry("l", late, list(range(len(late)))), StepEntry("o", other[pos_o: pos_o + 1], [0])])
    assert_close(out[: len(late)], want["l"], tol, "the newcomer")
    pos_o += 1
    assert set(held) & {p for p in runner.manager.block_table("l", 0) if p >= 0}, "pages were expected to be reused"
    runner.finish("l")
    # second pass: from position 0, portions of 13, the other request decoding beside it
    pos, again = 0, []
    while pos < len(victim):
        m = min(13, len(victim) - pos)
        entries = [StepEntry("v", victim[pos: pos + m], list(range(m)))]
        if pos_o < len(other):
            entries.append(StepEntry("o", other[pos_o: pos_o + 1], [0]))
        out = runner.step(entries)
        again.append(out[:m])
        if len(entries) == 2:
            assert_close(out[m:], want["o"][pos_o: pos_o + 1], tol, "the other request, second pass")
            pos_o += 1
        pos += m
    again = torch.cat(again)
    assert not torch.isnan(again).any()
    assert_close(again, want["v"], tol, "the request recomputed")
    if dtype == "float32":
        assert torch.equal(again[: first + 6], torch.cat(got)), "recomputation differs from the first pass"
    runner.manager.check()


def test_a_wait_that_runs_out_is_reported_and_leaves_the_engine_usable():
    """A kernel waits, with the wait that all tensor-core and bulk-copy kernels share, on a barrier
    that nobody completes; after a few hundred tries it gives up, leaves its code in the status
    word and returns.  The host sees it, the word is cleared, and the next step is right."""
    from mini_gpt_inference_b200.kernels.library import KernelLibraryError

    cfg, tensors, runner, tol = _setup("A", "bfloat16", False)
    ops = runner.ops
    ops.check_status()                                   # clean before
    ops.wait_probe(300)
    with pytest.raises(KernelLibraryError, match="gave up waiting \\(code 90\\)"):
        ops.check_status()
    ops.check_status()                                   # cleared by the report
    with pytest.raises(KernelLibraryError, match="limit"):
        ops.wait_probe(0)
    tokens = tokens_for(cfg, 40, 2)
    got = runner.step([StepEntry("r", tokens, list(range(40)))])
    assert_close(got, plain_logits(cfg, tensors, tokens), tol, "a step after the probe")
    ops.check_status()
