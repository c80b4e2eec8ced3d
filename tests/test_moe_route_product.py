"""Routing of many rows as a product and a selection (moe.cu, gemm_f32_tc5.cu): float32 prompts as one batch against the same
prompts one at a time, which route inside their norm kernel, and some of them against the oracle."""
from dataclasses import replace

import pytest

from helpers import C, W, make_oracle, rel_err
import nvllm_pkg

pytestmark = pytest.mark.gpu

SELECT_KERNEL = 52  # its id in the timeline


@pytest.mark.parametrize("experts,k,hidden,n,taken", [
    (8, 2, 264, 84, True),      # a quarter of a warp's lanes; k off the product's stages; rows off the tiles of 32
    (32, 8, 512, 84, True),     # all lanes
    (32, 8, 512, 80, False),    # fewer than 4096 rows
    (32, 8, 2048, 24, True),    # of wide ones
    (40, 5, 2048, 56, True),    # more experts than lanes, two tiles of them
    (130, 3, 1032, 36, True),   # three
    (40, 5, 264, 84, False),    # too little work
    (256, 4, 2048, 24, False),  # more than the selection has room for
])
def test_batch_matches_prompts_one_at_a_time(experts, k, hidden, n, taken):
    cfg = replace(C.tiny_granite(hidden=hidden, num_layers=2, ffn_dim=64), num_experts=experts, num_experts_per_tok=k)
    prompts = [W.random_prompt(cfg.vocab_size, 30 + (7 * i) % 41, 60 + i) for i in range(n)]  # some 50 rows each
    weights = list(W.random_weights(cfg, 3))
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, weights, precision=C.PREC_FP32, num_kv_blocks=n, sampling=None)

    def step(which):
        run.trace_begin(1 << 18)
        _, logits = run.run_flat([prompts[i] for i in which], True, [0] * len(which), [[i] for i in which], [0.0] * len(which),
                                 want_logits=True)
        return logits, SELECT_KERNEL in run.trace_end(1 << 18)[:, 1]

    try:
        batch, ran = step(range(n))
        assert ran == taken
        for i in range(0, n, 4):
            one, ran = step([i])
            assert not ran
            assert rel_err(batch[i], one[0]) <= 1e-4  # what the fp32 mode is held to against the reference
    finally:
        run.close()
    if taken and hidden <= 1032:
        oracle = make_oracle(cfg, 3)
        for i in (0, n // 2, n - 1):
            assert rel_err(batch[i], oracle.greedy(prompts[i], 1)[1][0]) <= 1e-4
