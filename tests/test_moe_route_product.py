"""Routing of many rows as a product and a selection (moe.cu, gemm_f32_tc5.cu): float32 prompts as one batch against the same
prompts one at a time, which route inside their norm kernel."""
from dataclasses import replace

import pytest

from helpers import C, W, rel_err
import nvllm_pkg

pytestmark = pytest.mark.gpu

SELECT_KERNEL = 52  # its id in the timeline


@pytest.mark.parametrize("experts,k,hidden,taken", [
    (8, 2, 264, True),      # a quarter of a warp's lanes; k off the product's stages
    (32, 8, 512, True),     # all lanes
    (40, 5, 264, True),     # more experts than lanes, two tiles of them
    (130, 3, 128, True),    # three
    (256, 4, 128, False),   # more than the selection has room for
])
def test_batch_matches_prompts_one_at_a_time(experts, k, hidden, taken):
    cfg = replace(C.tiny_granite(hidden=hidden, num_layers=2, ffn_dim=64), num_experts=experts, num_experts_per_tok=k)
    n = 24
    prompts = [W.random_prompt(cfg.vocab_size, 30 + (7 * i) % 41, 60 + i) for i in range(n)]  # 1200 rows: 38 tiles of 32
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, W.random_weights(cfg, 3), precision=C.PREC_FP32, num_kv_blocks=n, sampling=None)

    def step(which):
        run.trace_begin(1 << 18)
        _, logits = run.run_flat([prompts[i] for i in which], True, [0] * len(which), [[i] for i in which], [0.0] * len(which),
                                 want_logits=True)
        return logits, SELECT_KERNEL in run.trace_end(1 << 18)[:, 1]

    try:
        batch, ran = step(range(n))
        assert ran == taken
        for i in range(n):
            one, ran = step([i])
            assert not ran
            assert rel_err(batch[i], one[0]) <= 1e-4  # what the fp32 mode is held to against the reference
    finally:
        run.close()
