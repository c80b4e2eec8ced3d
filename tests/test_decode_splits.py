"""Decode attention on both sides of the lines where a context is left whole or split over CTAs (attention.cu
attn_decode_splits) and where a CTA takes two heads (attention_dec.cu): a decode step against the same tokens as ends of prompts."""
import numpy as np
import pytest

from helpers import C, W
import nvllm_pkg

pytestmark = pytest.mark.gpu

COMBINE = 14  # id in the timeline of the kernel that joins the parts


def gpt2():
    return C.tiny_gpt2(hidden=128, num_layers=2, num_heads=2, num_kv_heads=2, head_dim=64, ffn_dim=256, max_seq_len=2048)


def llama(kv):
    return C.tiny_llama(hidden=128, num_layers=2, num_heads=2 * kv, num_kv_heads=kv, head_dim=64, ffn_dim=256, max_seq_len=2048)


def falcon():
    return C.tiny_falcon(hidden=128, num_layers=2, num_heads=9, head_dim=64, ffn_dim=256, max_seq_len=2048)


@pytest.mark.parametrize("make,n,longest,split", [
    (gpt2, 1, 63, False), (gpt2, 3, 256, False), (gpt2, 2, 257, False),       # two heads to a CTA; one
    (gpt2, 2, 352, False), (gpt2, 2, 353, True),                              # few CTAs
    (lambda: llama(2), 27, 352, False), (lambda: llama(2), 27, 353, True),    # 54 CTAs
    (lambda: llama(2), 28, 353, False),                                       # 56
    (lambda: llama(8), 7, 1120, False), (lambda: llama(8), 7, 1121, True),    # 56 CTAs: 20 tokens each
    (falcon, 2, 256, False), (falcon, 2, 257, True),                          # one group of nine heads
], ids=lambda v: v if not callable(v) else "m")
def test_step_matches_the_prompts(make, n, longest, split):
    check_step(make(), [longest - (7 * i) % 31 for i in range(n)], split)


@pytest.mark.parametrize("rest,split", [(60, True), (1699, False)])
def test_one_long_context_among_short_ones(rest, split):
    """128 CTAs leave contexts whole where all are long, not where one is: the others' memory time does not hide it then."""
    check_step(llama(8), [1700] + [rest - (7 * i) % 31 for i in range(15)], split)


def check_step(cfg, lengths, split):
    n, longest = len(lengths), lengths[0]
    texts = [W.random_prompt(cfg.vocab_size, k, 160 + i) for i, k in enumerate(lengths)]
    weights = list(W.random_weights(cfg, 17, round_bf16=True))
    blocks = -(-longest // 256)
    tables, zeros = [list(range(blocks * i, blocks * i + blocks)) for i in range(n)], [0.0] * n

    def ends(precision, step):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, weights, precision=precision, num_kv_blocks=n * blocks, sampling=None)
        try:
            run.set_graphs(False)
            run.set_speculation(False)
            if not step:
                return run.run_flat(texts, True, [0] * n, tables, zeros, want_logits=True)[1]
            run.run_flat([t[:-1] for t in texts], True, [0] * n, tables, zeros)
            run.trace_begin(1 << 18)
            out = run.run_flat(texts, False, None, tables, zeros, want_logits=True)[1]
            assert (COMBINE in run.trace_end(1 << 18)[:, 1]) == split
            return out
        finally:
            run.close()

    want, prompts, step = ends(C.PREC_FP32, False), ends(C.PREC_BF16, False), ends(C.PREC_BF16, True)
    # the same bf16 roundings, sums in another order: as far from float32 as the prompts are; one row's error is known to
    # a third or so, that of n rows to the square root of n better
    assert np.linalg.norm(step - want) <= (1.2 + 0.4 / np.sqrt(n)) * np.linalg.norm(prompts - want)


def test_replayed_steps_choose_by_their_own_lengths():
    """Block tables with room to spare, so that nothing else of a step's shape changes where its kernels do: replayed steps give
    what launched ones give, bit for bit, whatever lengths the handle saw before."""
    cfg = gpt2()
    weights = list(W.random_weights(cfg, 17, round_bf16=True))
    texts = [W.random_prompt(cfg.vocab_size, n, 160 + i).tolist() for i, n in enumerate((250, 341, 30))]

    def drive(graphs):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, weights, precision=C.PREC_BF16, num_kv_blocks=6, sampling=None)
        try:
            run.set_graphs(graphs)
            run.set_speculation(False)
            outs, used = [], 0

            def steps(i, n):
                nonlocal used
                for k in range(n):
                    seq = texts[i] + [7 + j for j in range(k)]
                    outs.append(run.run_flat([seq], False, None, [[2 * i, 2 * i + 1]], [0.0], want_logits=True)[1])
                    used += run.last_stats.used_graph

            run.run_flat([t[:-1] for t in texts], True, [0] * 3, [[0, 1], [2, 3], [4, 5]], [0.0] * 3)
            steps(0, 12)  # across 256 tokens
            steps(2, 2)   # a short context after long ones
            steps(1, 14)  # a long one after short ones, across 352
            run.run_flat([texts[0]], False, None, [[0, 1]], [0.0])
            for _ in range(12):  # the same on the device's own tokens
                run.run_resident()
                used += run.last_stats.used_graph
                outs.append(run.sync(1)[0])
            return outs, used
        finally:
            run.close()

    (want, none), (got, all_) = drive(False), drive(True)
    assert none == 0 and all_ == len(got)
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)
