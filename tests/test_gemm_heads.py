"""The projections of an attention layer placed by the product's own epilogue (gemm_tc5_pair.cu): a batch of prompts that takes
it against the same prompts one at a time, whose heads are rotated and placed by a kernel of their own, and against the oracle."""
import numpy as np
import pytest

from helpers import C, W, make_oracle, rel_err
import nvllm_pkg

pytestmark = pytest.mark.gpu

ROPE_KERNEL, PAIR_KERNEL = 3, 46  # their ids in the timeline

FAMILIES = {
    # heads of 64: eight tiles of 128 columns with half of the last one empty, grouped keys; rotated, rows scaled by the folded norm
    "rope64": lambda: C.tiny_llama(hidden=520, num_layers=2, num_heads=9, num_kv_heads=3, head_dim=64, ffn_dim=512),
    "rope128": lambda: C.tiny_llama(hidden=520, num_layers=2, num_heads=17, num_kv_heads=1, head_dim=128, ffn_dim=512),
    # biases, no rotation, as many key heads as query heads
    "bias": lambda: C.tiny_gpt2(hidden=576, num_layers=2, num_heads=9, num_kv_heads=9, head_dim=64, ffn_dim=512),
    # one key head, a product beside the feed-forward
    "mqa": lambda: C.tiny_falcon(hidden=576, num_layers=2, num_heads=9, head_dim=64, ffn_dim=512),
}


@pytest.mark.parametrize("family", list(FAMILIES))
def test_batch_matches_prompts_one_at_a_time(family):
    cfg = FAMILIES[family]()
    # some 4400 rows of odd lengths, one prompt over the end of a page, one found half cached
    lens = [257] + [40 + (13 * i) % 97 for i in range(48)]
    prompts = [W.random_prompt(cfg.vocab_size, k, 60 + i) for i, k in enumerate(lens)]
    n = len(lens)
    tables = [[n, 0]] + [[i] for i in range(1, n)]
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, W.random_weights(cfg, 7, round_bf16=True), precision=C.PREC_BF16,
                                                  num_kv_blocks=n + 1, sampling=None)

    def step(which, cached):
        run.trace_begin(1 << 18)
        _, logits = run.run_flat([prompts[i] for i in which], True, cached, [tables[i] for i in which], [0.0] * len(which),
                                 want_logits=True)
        rec = run.trace_end(1 << 18)
        return logits, ROPE_KERNEL in rec[:, 1], PAIR_KERNEL in rec[:, 1]

    oracle = make_oracle(cfg, 7, round_bf16=True)
    exact = {i: oracle.greedy(prompts[i], 1)[1][0] for i in (0, 1, 24, n - 1)}
    try:
        alone = []
        for i in range(n):
            logits, rope, _ = step([i], [0])
            assert rope
            alone.append(logits[0])
        for cached in ([0] * n, [200] + [0] * (n - 1)):
            batch, rope, pair = step(range(n), cached)
            assert pair and not rope
            for i in range(n):
                # the same bf16 roundings, sums in another order: an element may round the other way (2^-8 of it)
                rms = np.sqrt(np.mean((batch[i] - alone[i]) ** 2) / np.mean(alone[i] ** 2))
                assert rms <= 1e-2, f"sequence {i}: {rms}"
            for i, want in exact.items():
                assert rel_err(batch[i], want) <= 2e-2  # what the bf16 mode is held to
    finally:
        run.close()
