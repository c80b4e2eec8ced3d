"""The two-CTA GEMM tiles of steps with many rows (gemm_tc5_pair.cu): the plain product against float64 torch at the
edges of its tiles, and every epilogue through whole steps — a batch of prompts that takes those tiles
against the same prompts one at a time, which do not; the device timeline says which kernel ran."""
from dataclasses import replace

import numpy as np
import pytest

from helpers import C, W
from test_gemm_tiles import _product
import nvllm_pkg
import test_zozonex as zozonex

pytestmark = pytest.mark.gpu

PAIR_KERNEL = 46  # its id in the timeline; a record's last word is the epilogue
PARTIAL, SWIGLU, GELU, RESID, RELU2 = range(5)


def _traced(run, call):
    """What the call returns, and the epilogues that the pair kernel ran with (the timeline is the process's own)."""
    run.trace_begin(1 << 18)
    out = call()
    rec = run.trace_end(1 << 18)
    assert 0 < len(rec) < 1 << 18
    return out, set(rec[rec[:, 1] == PAIR_KERNEL, 7].tolist())


@pytest.mark.parametrize("M,N,K,pair", [
    (257, 40000, 768, True),     # one row in the second token tile
    (512, 20000, 840, True),     # k tail, N off the tiles
    (520, 12928, 776, True),     # the last pair's second half lies outside W
    (1000, 10240, 1096, True),
    (300, 37901, 776, True),     # the last columns fill 13 lanes of a warp
    (300, 9216, 3072, True),     # one round
    (300, 9216, 3064, False),    # one round, less k
    (257, 40000, 760, False),    # several, less k
    (1100, 26496, 768, False),   # eight rounds instead of seven
])
def test_pair_product(M, N, K, pair):
    R = nvllm_pkg.sub("runner")
    cfg = C.tiny_gpt2()
    run = R.CudaModelRunner(cfg, W.random_weights(cfg, 1), num_kv_blocks=1, sampling=None)
    try:
        error, ran = _traced(run, lambda: _product(M, N, K, C.PREC_BF16, 3))
    finally:
        run.close()
    assert error <= 1.0
    assert ran == ({PARTIAL} if pair else set())


def _family(family):
    if family.startswith("k="):  # one k block; four, fewer than the stages, with a tail
        k = int(family[2:])
        return C.tiny_llama(hidden=k, num_layers=2, num_heads=3, num_kv_heads=1, head_dim=64, ffn_dim=2048), {SWIGLU}
    if family == "rms_swiglu_resid":  # 18 x 17 tiles of the residual products, 24 lanes of a warp in the last columns
        return C.tiny_llama(hidden=2200, num_layers=2, num_heads=34, num_kv_heads=2, head_dim=64, ffn_dim=2048), {PARTIAL, SWIGLU, RESID}
    if family == "gelu":
        return C.tiny_falcon(hidden=1024, num_layers=2, num_heads=16, head_dim=64, ffn_dim=8200), {GELU}
    if family == "moe":  # all experts chosen: rounding cannot flip a choice
        return replace(C.tiny_granite(hidden=1024, num_layers=2, num_heads=16, num_kv_heads=4, head_dim=64, ffn_dim=768),
                       num_experts=8, num_experts_per_tok=8), {PARTIAL, SWIGLU}
    return zozonex.model([zozonex.layer(zozonex.attn(heads=4, kv_heads=2, dim=64, vdim=64, window=60), 8200)] * 2, width=1024), {RELU2}


@pytest.mark.parametrize("family", ["rms_swiglu_resid", "gelu", "relu2", "moe", "k=64", "k=200"])
def test_batch_matches_prompts_one_at_a_time(family):
    R = nvllm_pkg.sub("runner")
    cfg, epilogues = _family(family)
    if isinstance(cfg, dict):
        cfg, w = zozonex.random_weights(cfg, 7, bf16=True)
        weights = w.items()
    else:
        weights = W.random_weights(cfg, 7, round_bf16=True)
    n, lens = 46, [80 + (7 * i) % 23 for i in range(46)]  # 4177 rows
    prompts = [W.random_prompt(cfg.vocab_size, k, 60 + i) for i, k in enumerate(lens)]
    run = R.CudaModelRunner(cfg, weights, precision=C.PREC_BF16, num_kv_blocks=n, sampling=None)
    try:
        (_, batch), ran = _traced(run, lambda: run.run_flat(prompts, True, [0] * n, [[i] for i in range(n)], [0.0] * n, want_logits=True))
        assert ran >= epilogues
        for i in range(n):
            (_, one), ran = _traced(run, lambda: run.run_flat([prompts[i]], True, [0], [[i]], [0.0], want_logits=True))
            assert not ran
            # the same bf16 roundings, sums in another order: an element may round the other way (2^-8 of it)
            rms = np.sqrt(np.mean((batch[i] - one[0]) ** 2) / np.mean(one[0] ** 2))
            assert rms <= 1e-2, f"sequence {i}: {rms}"
    finally:
        run.close()
