"""The two-CTA GEMM tiles of steps with many rows (gemm_tc5_pair.cu): the plain product against float64 torch at the
edges of its tiles, and every epilogue through whole steps — a batch of prompts that takes those tiles
against the same prompts one at a time, which do not."""
from dataclasses import replace

import numpy as np
import pytest

from helpers import C, W
from test_gemm_tiles import _product
import nvllm_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [
    (257, 40000, 64),    # one k block, one row in the second token tile
    (512, 20000, 200),   # k tail, N off the tiles
    (520, 12928, 136),   # the last pair's second half lies outside W
    (1000, 10240, 456),  # more k blocks than stages
    (300, 37901, 72),    # the last columns fill 13 lanes of a warp
])
def test_pair_product(M, N, K):
    assert _product(M, N, K, C.PREC_BF16, 3) <= 1.0


@pytest.mark.parametrize("family", ["rms_swiglu_resid", "gelu", "moe"])
def test_batch_matches_prompts_one_at_a_time(family):
    R = nvllm_pkg.sub("runner")
    if family == "rms_swiglu_resid":
        cfg = C.tiny_llama(hidden=2048, num_layers=2, num_heads=32, num_kv_heads=8, head_dim=64, ffn_dim=2048)
    elif family == "gelu":
        cfg = C.tiny_falcon(hidden=1024, num_layers=2, num_heads=16, head_dim=64, ffn_dim=8192)
    else:
        cfg = replace(C.tiny_granite(hidden=1024, num_layers=2, num_heads=16, num_kv_heads=4, head_dim=64, ffn_dim=512),
                      num_experts=8, num_experts_per_tok=8)  # all experts chosen: rounding cannot flip a choice
    n, lens = 20, [130 + (7 * i) % 23 for i in range(20)]
    prompts = [W.random_prompt(cfg.vocab_size, k, 60 + i) for i, k in enumerate(lens)]
    run = R.CudaModelRunner(cfg, W.random_weights(cfg, 7, round_bf16=True), precision=C.PREC_BF16, num_kv_blocks=n, sampling=None)
    try:
        _, batch = run.run_flat(prompts, True, [0] * n, [[i] for i in range(n)], [0.0] * n, want_logits=True)
        for i in range(n):
            _, one = run.run_flat([prompts[i]], True, [0], [[i]], [0.0], want_logits=True)
            # the same bf16 roundings, sums in another order: an element may round the other way (2^-8 of it)
            rms = np.sqrt(np.mean((batch[i] - one[0]) ** 2) / np.mean(one[0] ** 2))
            assert rms <= 1e-2, f"sequence {i}: {rms}"
    finally:
        run.close()
