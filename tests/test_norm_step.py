"""Norms of steps of few rows (elementwise.cu norm_rows_kernel, slices of a product summed on the way): a decode step against
the same tokens as the ends of whole prompts, whose norms are other kernels or part of the products."""
import numpy as np
import pytest

from helpers import C, W
import nvllm_pkg

pytestmark = pytest.mark.gpu

ROWS, GENERAL = 53, 2  # kernel ids in the timeline


def gpt2(hidden):
    return C.tiny_gpt2(hidden=hidden, num_layers=2, num_heads=2, num_kv_heads=2, head_dim=64, ffn_dim=1096)


def llama(hidden):
    return C.tiny_llama(hidden=hidden, num_layers=2, num_heads=4, num_kv_heads=2, head_dim=64, ffn_dim=1096)


def falcon(hidden):
    return C.tiny_falcon(hidden=hidden, num_layers=2, num_heads=3, head_dim=64, ffn_dim=1096)


@pytest.mark.parametrize("cfg", [
    gpt2(64), llama(72),                       # half a warp; a thread more
    gpt2(2056), llama(2560), falcon(2048),     # one vector, the last one: five slices and more
    llama(2568), falcon(4544), gpt2(5120),     # two
    falcon(5128), llama(7688),                 # three; four
    llama(6144), falcon(6152), gpt2(8192), llama(8200),  # the last of three, of four; five
    gpt2(10240), llama(10248),                 # the widest; wider
], ids=lambda c: f"{c.name}-{c.hidden}")
def test_step_matches_the_prompts(cfg):
    check_step(cfg, [61 + 3 * i for i in range(12)], cfg.hidden <= 10240)


@pytest.mark.parametrize("cfg,n,rows", [
    (llama(2048), 444, True), (llama(2048), 445, False),    # three waves, one CTA to an SM
    (llama(2056), 511, True),                               # norm_kernel has no more of them there
    (gpt2(8192), 148, True), (gpt2(8192), 149, False),      # four vectors: one wave
], ids=lambda v: v.hidden if hasattr(v, "hidden") else str(v))
def test_wide_batches(cfg, n, rows):
    check_step(cfg, [2 + i % 3 for i in range(n)], rows)


def check_step(cfg, lengths, rows):
    n = len(lengths)
    texts = [W.random_prompt(cfg.vocab_size, k, 160 + i) for i, k in enumerate(lengths)]
    weights = list(W.random_weights(cfg, 17, round_bf16=True))
    tables, zeros = [[i] for i in range(n)], [0.0] * n

    def ends(precision, step):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, weights, precision=precision, num_kv_blocks=n, sampling=None)
        try:
            run.set_graphs(False)
            run.set_speculation(False)
            if not step:
                return run.run_flat(texts, True, [0] * n, tables, zeros, want_logits=True)[1]
            run.run_flat([t[:-1] for t in texts], True, [0] * n, tables, zeros)
            run.trace_begin(1 << 18)
            out = run.run_flat(texts, False, None, tables, zeros, want_logits=True)[1]
            ran = set(run.trace_end(1 << 18)[:, 1].tolist())
            assert (ROWS in ran, GENERAL in ran) == (rows, not rows)
            return out
        finally:
            run.close()

    want, prompts, step = ends(C.PREC_FP32, False), ends(C.PREC_BF16, False), ends(C.PREC_BF16, True)
    # the same bf16 roundings, sums in another order: as far from float32 as the prompts are (the error's norm over n rows is
    # known to a tenth or so)
    assert np.linalg.norm(step - want) <= 1.25 * np.linalg.norm(prompts - want)


@pytest.mark.parametrize("cfg", [C.tiny_llama(hidden=24), falcon(64), C.tiny_granite(hidden=264)], ids=lambda c: c.name)
def test_rows_asked_for_twice(cfg):
    """The logits of rows that are a sequence's last one as well: the last norm meets them twice, and takes their pending results
    in each time from the same residual row."""
    n = 24
    texts = [W.random_prompt(cfg.vocab_size, 3 + i % 5, 60 + i) for i in range(n)]
    last = (np.cumsum([len(t) for t in texts]) - 1).tolist()
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, W.random_weights(cfg, 3), precision=C.PREC_FP32, num_kv_blocks=n, sampling=None)
    try:
        for _ in range(40):
            run.request_logits(last + last)
            _, once = run.run_flat(texts, True, [0] * n, [[i] for i in range(n)], [0.0] * n, want_logits=True)
            again = run.fetch_logits(2 * n)
            np.testing.assert_array_equal(again[:n], once)
            np.testing.assert_array_equal(again[n:], once)
    finally:
        run.close()
