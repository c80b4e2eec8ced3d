"""Routing and sorting of steps of few rows (elementwise.cu norm_route_kernel, moe.cu moe_sort_gather_kernel): a decode step
against the same tokens as the ends of whole prompts of more than 1024 rows, which other kernels route and sort."""
import numpy as np
import pytest

from helpers import C, W
import nvllm_pkg

pytestmark = pytest.mark.gpu

ROUTE, SORT = 54, 17  # kernel ids in the timeline


@pytest.mark.parametrize("hidden,experts,k,n", [
    (64, 3, 2, 12),        # fewer experts than warps, half a piece
    (72, 17, 4, 12),       # one warp with two experts
    (1024, 32, 8, 128),    # all of the router's rows ahead of the wait; one chunk of pairs
    (1032, 33, 8, 130),    # a ninth piece; more experts than lanes; two chunks
    (2056, 64, 3, 40),     # two vectors a row
    (520, 64, 16, 256),    # four chunks of pairs, the most that are sorted at once
    (264, 96, 9, 30),      # more experts than are sorted at once
])
def test_step_matches_the_prompts(hidden, experts, k, n):
    cfg = C.tiny_granite(hidden=hidden, num_experts=experts, num_experts_per_tok=k, ffn_dim=64, num_layers=2)
    long = -(-1100 // n) + 8
    texts = [W.random_prompt(cfg.vocab_size, long + i % 7, 160 + i) for i in range(n)]
    weights = list(W.random_weights(cfg, 17, round_bf16=True))
    tables, zeros = [[i] for i in range(n)], [0.0] * n

    def ends(precision, step):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, weights, precision=precision, num_kv_blocks=n, sampling=None)
        try:
            run.set_graphs(False)
            run.set_speculation(False)
            if step:
                run.run_flat([t[:-1] for t in texts], True, [0] * n, tables, zeros)
            run.trace_begin(1 << 18)
            out = run.run_flat(texts, not step, [0] * n if not step else None, tables, zeros, want_logits=True)[1]
            ran = set(run.trace_end(1 << 18)[:, 1].tolist())
            assert (ROUTE in ran) == step
            if precision == C.PREC_BF16 and step:
                assert (SORT in ran) == (experts <= 64 and n * k <= 4096)
            return out
        finally:
            run.close()

    want, step = ends(C.PREC_FP32, False), ends(C.PREC_FP32, True)
    # what the fp32 mode is held to against the reference
    assert np.abs(step - want).max() <= 1e-4 * np.abs(want).max()
    # bf16: the same roundings, sums in another order; a choice between two experts may fall the other way in either
    prompts, step = ends(C.PREC_BF16, False), ends(C.PREC_BF16, True)
    assert np.linalg.norm(step - want) <= 1.25 * np.linalg.norm(prompts - want)
