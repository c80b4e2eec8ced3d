"""The speculative next step of nvllm_run: calls that never ask for it pause it, a decode loop gets it back, and results (tokens,
logits, device time of the step that was asked for) are those of a runner without it."""
import importlib

import numpy as np
import pytest

from helpers import C, W
import nvllm_pkg
import test_zozonex as zozonex

pytestmark = pytest.mark.gpu


def test_prompts_pause_it_and_decoding_brings_it_back():
    cfg = C.tiny_llama()
    prompts = [W.random_prompt(cfg.vocab_size, 18 + 7 * i, 300 + i).tolist() for i in range(3)]
    tables = [[i] for i in range(3)]

    def drive(spec):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, W.random_weights(cfg, 5), precision=C.PREC_FP32, num_kv_blocks=3, sampling=None)
        try:
            run.set_speculation(spec)
            outs, hits = [], []
            for _ in range(12):  # each call after a speculation is a miss; the pauses grow to 16 calls
                outs.append(run.run_flat(prompts, True, [0] * 3, tables, [0.0] * 3, want_logits=True))
            seqs = [list(p) for p in prompts]
            for k in range(40):
                for s, t in zip(seqs, outs[-1][0]):
                    s.append(int(t))
                outs.append(run.run_flat(seqs, False, None, tables, [0.0] * 3, want_logits=k % 2 == 0))
                hits.append(run.last_stats.h2d_bytes == 0)
                assert run.last_stats.device_ms > 0
            return outs, hits
        finally:
            run.close()

    (want, none), (got, hits) = drive(False), drive(True)
    assert not any(none)
    first = hits.index(True)
    assert first <= 17 and all(hits[first:])
    for (a, la), (b, lb) in zip(want, got):
        np.testing.assert_array_equal(a, b)
        assert (la is None) == (lb is None)
        if la is not None:
            np.testing.assert_array_equal(la, lb)  # same kernels, same order


def test_arrivals_discard_one_step_each():
    """Prompts that arrive while others decode: each costs the step that was issued for the batch without it, and the steps
    issued behind the prompts themselves, which the merged batch never asks for, die out."""
    cfg = C.tiny_llama()
    prompts = [W.random_prompt(cfg.vocab_size, 18 + 7 * i, 300 + i).tolist() for i in range(20)]
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, W.random_weights(cfg, 5), precision=C.PREC_FP32, num_kv_blocks=20, sampling=None)

    def call(which, prefill, hit=None):
        nonlocal issued
        seqs = [prompts[i] for i in which]
        out, _ = run.run_flat(seqs, prefill, [0] * len(seqs), [[i] for i in which], [0.0] * len(seqs))
        if hit is not None:
            assert (run.last_stats.h2d_bytes == 0) == hit, (which, hit)
        issued = run.sync()[1] != run.last_stats.device_ms  # the time of the last step issued is not that of the one asked for
        for s, t in zip(seqs, out):
            s.append(int(t))

    issued, live = False, [0, 1, 2]
    try:
        call(live, True)
        for _ in range(3):
            call(live, False, hit=True)
        for arrival in range(3, 20):
            call([arrival], True, hit=False)
            if arrival - 3 not in (0, 2, 5, 10):  # pauses of 1, 2, 4 and 8 prompts
                assert not issued, arrival
            live = live[1:] + [arrival]
            call(live, False, hit=False)
            for _ in range(3):  # the merged batch goes on without the host at once
                call(live, False, hit=True)
    finally:
        run.close()


def test_recurrent_state_of_steps_that_are_not_asked_for():
    """Calls that a step issued ahead does not match (another token, another batch), on a model whose steps update state in
    place: the same with steps issued ahead, whose state is put back, as without."""
    cfg, w = zozonex.random_weights(zozonex.mixed_model(), 7)
    prompts = [W.random_prompt(cfg.vocab_size, 9 + 4 * i, 40 + i).tolist() for i in range(3)]

    def drive(spec):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, w.items(), precision=C.PREC_FP32, num_kv_blocks=3, sampling=None, num_state_slots=3)
        try:
            run.set_speculation(spec)
            seqs = [list(p) for p in prompts]
            outs = [run.run_flat(seqs, True, [0] * 3, [[0], [1], [2]], [0.0] * 3, want_logits=True, state_slots=[2, 0, 1])]
            for k in range(8):
                for i, (s, t) in enumerate(zip(seqs, outs[-1][0])):
                    s.append(5 if (k, i) == (2, 1) else int(t))
                if k == 5:  # the first sequence alone, before all three
                    outs.append(run.run_flat(seqs[:1], False, None, [[0]], [0.0], want_logits=True, state_slots=[2]))
                    seqs[0].append(int(outs[-1][0][0]))
                outs.append(run.run_flat(seqs, False, None, [[0], [1], [2]], [0.0] * 3, want_logits=True, state_slots=[2, 0, 1]))
            return outs
        finally:
            run.close()

    for (a, la), (b, lb) in zip(drive(False), drive(True)):
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(la, lb)


@pytest.mark.parametrize("family", ["zozonex", "lazovik", "sutuvik", "sozurax", "defilorn"])
def test_recurrent_state_goes_back(family):
    """Steps issued ahead on models whose steps update state in place: taken where they match; where the next call has another
    token, batch, order or slots, or is a prompt, the state they changed is put back."""
    m = importlib.import_module("test_" + family)
    cfg, w = m.random_weights(m.mixed_model(), 7)
    prompts = [W.random_prompt(cfg.vocab_size, 9 + 4 * i, 40 + i).tolist() for i in range(4)]

    def drive(spec):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, w.items(), precision=C.PREC_FP32, num_kv_blocks=4, sampling=None, num_state_slots=5)
        try:
            run.set_speculation(spec)
            seqs, slots, outs, hits = [list(p) for p in prompts], [2, 0, 1, 4], [], 0

            def call(which, prompt=False):
                nonlocal hits
                out, logits = run.run_flat([seqs[i] for i in which], prompt, [0] * len(which), [[i] for i in which], [0.0] * len(which),
                                           want_logits=True, state_slots=[slots[i] for i in which])
                hits += run.last_stats.h2d_bytes == 0
                outs.append((out, logits))
                for i, t in zip(which, out):
                    seqs[i].append(int(t))

            call([0, 1, 2], prompt=True)
            for k in range(24):
                if k in (3, 15):
                    seqs[1][-1] = 5  # another token than the one that came out
                if k == 6:
                    call([0])        # one of them alone
                if k == 9:
                    call([2, 0, 1])  # another order
                if k == 12:          # a new sequence joins; one ends and its slot is the next one's
                    call([3], prompt=True)
                if k == 18:
                    seqs[3], slots[3] = list(prompts[3]), 3
                    call([3], prompt=True)
                if k == 21:
                    run.sync()
                call([0, 1, 2])
            call([3])
            return outs, hits
        finally:
            run.close()

    (want, none), (got, hits) = drive(False), drive(True)
    assert none == 0 and hits >= 10
    for (a, la), (b, lb) in zip(want, got):
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(la, lb)


@pytest.mark.parametrize("family", ["zozonex", "lazovik", "sutuvik", "sozurax", "defilorn"])
def test_recurrent_state_in_repeated_and_resident_steps(family):
    """A repetition of a prompt step (rerun) puts the state back that the step in flight behind it changed; run_resident takes the
    step in flight, and the next call goes on from its state, whether it asks for the step after it or for another token."""
    m = importlib.import_module("test_" + family)
    cfg, w = m.random_weights(m.mixed_model(), 7)
    prompts = [W.random_prompt(cfg.vocab_size, 9 + 4 * i, 40 + i).tolist() for i in range(3)]

    def drive(spec):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, w.items(), precision=C.PREC_FP32, num_kv_blocks=3, sampling=None, num_state_slots=3)
        try:
            run.set_speculation(spec)
            seqs, outs, issued = [list(p) for p in prompts], [], 0

            def append(tokens):
                for s, t in zip(seqs, tokens):
                    s.append(int(t))

            def call(prompt=False):
                nonlocal issued
                out, logits = run.run_flat(seqs, prompt, [0] * 3, [[0], [1], [2]], [0.0] * 3, want_logits=True, state_slots=[2, 0, 1])
                outs.extend((out, logits))
                # the time of the last step issued is not that of the one asked for
                issued += run.sync()[1] != run.last_stats.device_ms
                append(out)

            def resident():
                run.run_resident()
                outs.append(run.sync(3)[0].copy())
                append(outs[-1])

            call(prompt=True)
            for _ in range(2):
                run.rerun()
                outs.append(run.sync(3)[0].copy())
            for k in range(12):
                call()
                if k in (2, 5, 8):
                    resident()
                if k == 5:
                    resident()       # one that is not in flight
                if k in (5, 8):
                    seqs[1][-1] = 5  # another token than the one that came out
            return outs, issued
        finally:
            run.close()

    (want, none), (got, issued) = drive(False), drive(True)
    assert none == 0 and issued >= 5
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,ahead", [(31, True), (32, False)])
def test_room_for_the_state(n, ahead):
    """4 MB of state a sequence: up to 128 MB are copied aside, a step of more waits for the host.  The room is made with the
    handle, not between decode steps, and is part of what memory_info says."""
    torch = pytest.importorskip("torch")
    z = zozonex
    cfg, w = z.random_weights(z.model([z.layer(z.delta(heads=64, kv_heads=8, dim=128, vdim=128, conv=2), 48),
                                       z.layer(z.attn(heads=2, kv_heads=1, dim=16, vdim=16, window=40))]), 7)
    prompts = [W.random_prompt(cfg.vocab_size, 3 + i % 3, 40 + i).tolist() for i in range(n)]

    def drive(spec):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, w.items(), precision=C.PREC_FP32, num_kv_blocks=n, sampling=None, num_state_slots=n)
        try:
            run.set_speculation(spec)
            seqs, outs, hits, start = [list(p) for p in prompts], [], 0, torch.cuda.mem_get_info()[0]

            def call(which, prompt, temperature):
                nonlocal hits
                out, logits = run.run_flat([seqs[i] for i in which], prompt, [0] * len(which), [[i] for i in which],
                                           [temperature] * len(which), [0.5] * len(which), want_logits=True, state_slots=list(which))
                hits += run.last_stats.h2d_bytes == 0
                outs.extend((out, logits))
                for i, t in zip(which, out):
                    seqs[i].append(int(t))

            call(range(n), True, 1.0)  # (nothing is issued behind a step with draws)
            free, room = torch.cuda.mem_get_info()[0], run.memory_info()["workspace"]
            for _ in range(4):
                call(range(2), False, 0.0)
            two = hits
            for _ in range(6):
                call(range(n), False, 0.0)
            end = torch.cuda.mem_get_info()[0]
            assert free - end < 16 << 20 and run.memory_info()["workspace"] == room  # (graphs)
            return outs, two, hits - two, start - end - room
        finally:
            run.close()

    (want, *none, beside), (got, two, hits, beside_ahead) = drive(False), drive(True)
    assert none == [0, 0] and two == 3 and hits == (5 if ahead else 0)
    assert beside_ahead - beside < 16 << 20
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)


def test_requested_logits_rows():
    """Further rows asked for (nvllm_request_logits) in calls that a step issued ahead would answer or overwrite."""
    cfg = C.tiny_llama(hidden=1032)  # the head's products of few rows are split along k: another step's slices are elsewhere
    prompts = [W.random_prompt(cfg.vocab_size, 18 + 7 * i, 300 + i).tolist() for i in range(3)]
    weights = list(W.random_weights(cfg, 5))

    def drive(spec):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, weights, precision=C.PREC_FP32, num_kv_blocks=3, sampling=None)
        try:
            run.set_speculation(spec)
            seqs, rows, outs, hits = [list(p) for p in prompts], [3, 20, 40, 7], [], 0
            for k in range(9):
                want = rows if k == 0 else [2, 0] if k in (4, 7) else []
                run.request_logits(want)
                out, logits = run.run_flat(seqs, k == 0, [0] * 3, [[0], [1], [2]], [0.0] * 3, want_logits=True)
                hits += run.last_stats.h2d_bytes == 0
                outs += [out, logits] + ([run.fetch_logits(len(want))] if want else [])
                for s, t in zip(seqs, out):
                    s.append(int(t))
            return outs, hits
        finally:
            run.close()

    (want, none), (got, hits) = drive(False), drive(True)
    assert none == 0 and hits >= 3
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)
