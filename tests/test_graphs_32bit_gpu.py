"""32-bit steps replayed as CUDA graphs: the same bits as the steps run eagerly, whatever shares the step, for every architecture;
what a step hands out stays as it is; which steps are captured, and when."""
import threading

import pytest
import torch

from odin_infer_b200 import Engine, Engine_Opts, StepEntry
from odin_infer_b200.config import config_from_dict
from tests import test_bafilorn_gpu, test_fugavik_gpu, test_meropel_gpu, test_nikonex_gpu, test_nufupel_gpu, test_tovalix_gpu, tiny
from tests.tiny import random_tokens

pytestmark = pytest.mark.gpu

MODELS = {"qwen3": tiny.TINY_D, "tovalix": test_tovalix_gpu.MIXED, "nufupel": test_nufupel_gpu.MIXED, "nikonex": test_nikonex_gpu.MIXED,
          "meropel": test_meropel_gpu.MIXED, "fugavik": test_fugavik_gpu.MIXED, "bafilorn": test_bafilorn_gpu.MIXED}


def engine_of(name, graphs=True, max_batch=4, max_ctx=512):
    return Engine.random(config_from_dict(MODELS[name]), 5, Engine_Opts(max_ctx=max_ctx, max_batch=max_batch, dtype="float32",
                                                                        verbose=False, cuda_graphs=graphs))


def prompts_of(engine, lens, seed):
    return [random_tokens(n, engine.vocab_size, seed + i) for i, n in enumerate(lens)]


def request(engine, prompts, steps=2):
    """The prompts in one step, the last place of each wanted, then `steps` steps of one token; the logits of every step,
    as the engine handed them out."""
    slots = [engine.take_slot() for _ in prompts]
    got = [engine.step([StepEntry(s, p, [len(p) - 1]) for s, p in zip(slots, prompts)])]
    for i in range(steps):
        got.append(engine.step([StepEntry(s, [7 + i], [0]) for s in slots]))
    for s in slots:
        engine.give_back_slot(s)
    return got


# Beside the lengths at which a recurrence changes its form (128 and 256 tokens) stand lengths whose buckets reach that line and
# they do not, alone and because of what shares the step.
@pytest.mark.parametrize("name", list(MODELS))
def test_replayed_steps_are_the_eager_steps_bit_for_bit(name):
    on, off = engine_of(name, True), engine_of(name, False)
    for lens in ((200,), (130, 100), (40, 40), (20,), (3, 9, 2), (65,), (127, 2), (128,), (255,), (256,), (100, 27, 128)):
        prompts = prompts_of(on, lens, 100)
        want = request(off, prompts)
        for turn in range(4):       # eagerly, captured, replayed twice
            for i, (a, b) in enumerate(zip(request(on, prompts), want)):
                assert torch.equal(a, b), (name, lens, turn, i, float((a - b).abs().max() / b.abs().max()))
    on.destroy(), off.destroy()


@pytest.mark.parametrize("name", list(MODELS))
def test_a_request_has_the_same_bits_alone_and_beside_others(name):
    """The lengths of a step lie on one side of the lines between a recurrence's forms, which the longest of them chooses."""
    engine = engine_of(name)
    for lens in ((120, 100) if name == "fugavik" else (130, 100), (40, 40), (20, 9), (90, 100, 30)):
        prompts = prompts_of(engine, lens, 200)
        alone = [request(engine, [p]) for p in prompts]
        for turn in range(4):
            for i, got in enumerate(request(engine, prompts)):
                for j in range(len(prompts)):
                    assert torch.equal(got[j:j + 1], alone[j][i]), (name, lens, turn, i, j)
    engine.destroy()


def graphs_of(engine):
    keys = engine.graphs._graphs
    return {k for k in keys if k[0] == "prompt"}, {k for k in keys if k[0] != "prompt"}


def test_a_decode_graph_serves_every_context_length():
    """Decoding from 500 to 530 tokens, across the border of what are two classes of contexts in bfloat16."""
    on, off = engine_of("qwen3", True, max_ctx=640), engine_of("qwen3", False, max_ctx=640)
    prompt = prompts_of(on, (500,), 300)
    for a, b in zip(request(on, prompt, 30), request(off, prompt, 30)):
        assert torch.equal(a, b)
    assert len(graphs_of(on)[1]) == 1
    on.destroy(), off.destroy()


def test_a_shape_of_step_is_captured_when_it_comes_again():
    """Prompts of lengths that come once run eagerly; the second step of a bucket is captured."""
    engine = engine_of("qwen3")
    for n in (10, 30, 60, 120):
        request(engine, prompts_of(engine, (n,), n), steps=0)
    assert graphs_of(engine) == (set(), set())
    request(engine, prompts_of(engine, (50,), 1), steps=1)
    prompts, decodes = graphs_of(engine)
    assert [k[1] for k in prompts] == [64] and not decodes
    request(engine, prompts_of(engine, (200,), 1), steps=1)
    prompts, decodes = graphs_of(engine)
    assert [k[1] for k in prompts] == [64] and [k[0] for k in decodes] == [1]
    engine.destroy()


def test_engines_in_several_threads_capture_side_by_side():
    """Three engines of the same weights, each in a thread of its own on a stream of its own, that allocate, copy and capture at
    the same time: no step fails, and all hand out the same logits.  (In 32-bit: two launches of bfloat16 attention must not
    overlap on a device, see the counters in its kernels.)"""
    engines = [engine_of("qwen3", max_ctx=320) for _ in range(3)]
    torch.cuda.synchronize()
    outs, errors = [[] for _ in engines], []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for n in (3, 20, 60, 130, 250):
                    for batch in (1, 2, 3):
                        prompts = [[1 + b] * max(2, n // batch) for b in range(batch)]
                        for turn in range(3):
                            outs[k] += [x.cpu() for x in request(engines[k], prompts)]
                            torch.full((1 << 20,), turn, device="cuda:0")
        except Exception as e:   # noqa: BLE001
            errors.append(repr(e))
    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for o in outs[1:]:
        assert len(o) == len(outs[0]) and all(torch.equal(a, b) for a, b in zip(o, outs[0]))
    for e in engines:
        e.destroy()


def test_a_capture_that_failed_leaves_the_engine_able_to_capture(monkeypatch):
    """The failure is made on the host, while the first capture is under way; the step raises, and the next ones are captured
    and replayed."""
    on, off = engine_of("qwen3", True), engine_of("qwen3", False)
    prompt = prompts_of(on, (20,), 400)
    want = request(off, prompt)
    request(on, prompt, steps=0)                    # eagerly
    run = on.rt.run
    calls = []

    def fails_while_capturing(model, batch):
        out = run(model, batch)
        calls.append(torch.cuda.is_current_stream_capturing())
        if calls[-1]:
            raise RuntimeError("made by the test")
        return out
    monkeypatch.setattr(on.rt, "run", fails_while_capturing)
    slot = on.take_slot()
    with pytest.raises(RuntimeError, match="made by the test"):
        on.step([StepEntry(slot, prompt[0], [19])])
    on.give_back_slot(slot)
    assert calls == [False, True] and graphs_of(on) == (set(), set())
    monkeypatch.setattr(on.rt, "run", run)
    for turn in range(3):
        for a, b in zip(request(on, prompt), want):
            assert torch.equal(a, b)
    assert all(graphs_of(on))
    on.destroy(), off.destroy()


def test_graphs_thrown_away_are_captured_anew():
    engine = engine_of("qwen3")
    prompt = prompts_of(engine, (20,), 400)
    first = request(engine, prompt)
    for turn in range(2):
        for again in range(3):
            assert all(torch.equal(a, b) for a, b in zip(request(engine, prompt), first))
        assert all(graphs_of(engine))
        engine.graphs.clear()
    engine.destroy()


def test_steps_that_want_several_places_of_a_sequence_run_eagerly():
    """Also where another sequence of the step wants none."""
    engine = engine_of("qwen3")
    for wants in (([3, 9], []), ([9], [0, 11])):
        for turn in range(3):
            slots = [engine.take_slot() for _ in wants]
            logits = engine.step([StepEntry(s, list(range(1, 13)), w) for s, w in zip(slots, wants)])
            assert len(logits) == sum(map(len, wants))
            for s in slots:
                engine.give_back_slot(s)
    assert not graphs_of(engine)[0]
    engine.destroy()


@pytest.mark.parametrize("name", ["qwen3", "fugavik", "meropel"])
def test_replays_that_share_a_pool_leave_one_another_and_what_was_handed_out_alone(name):
    """Graphs of several prompt and decode buckets, captured in one order and replayed in others: every step's logits are
    the eager step's, and those that a caller kept do not change under later replays."""
    on, off = engine_of(name, True), engine_of(name, False)
    groups = [(20,), (100, 27), (50, 9, 60), (200,), (5,)]
    prompts = [prompts_of(on, lens, 500 + 10 * i) for i, lens in enumerate(groups)]
    want = [request(off, p) for p in prompts]
    for turn in range(2):                          # seen, captured
        for p in prompts:
            request(on, p)
    captured = [set(keys) for keys in graphs_of(on)]
    assert len(captured[0]) == len(groups) and len(captured[1]) == 3
    kept = []
    for order in ([4, 0, 2, 1, 3], [3, 2, 1, 0, 4], [1, 1, 4, 4, 0]):
        for i in order:
            kept.append((i, request(on, prompts[i])))
    for i, got in kept:
        for a, b in zip(got, want[i]):
            assert torch.equal(a, b), (name, i)
    assert [set(keys) for keys in graphs_of(on)] == captured
    on.destroy(), off.destroy()
