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


@pytest.mark.parametrize("M,N,K", [
    (257, 40000, 64),    # one k block, one row in the second token tile
    (512, 20000, 200),   # k tail, N off the tiles
    (520, 12928, 136),   # the last pair's second half lies outside W
    (1000, 10240, 456),  # more k blocks than stages
    (300, 37901, 72),    # the last columns fill 13 lanes of a warp
])
def test_pair_product(M, N, K):
    assert _product(M, N, K, C.PREC_BF16, 3) <= 1.0


def _family(family):
    if family == "rms_swiglu_resid":  # 18 x 17 tiles of the residual products, 24 lanes of a warp in the last columns
        return C.tiny_llama(hidden=2200, num_layers=2, num_heads=34, num_kv_heads=2, head_dim=64, ffn_dim=2048), {PARTIAL, SWIGLU, RESID}
    if family == "gelu":
        return C.tiny_falcon(hidden=1024, num_layers=2, num_heads=16, head_dim=64, ffn_dim=8200), {GELU}
    if family == "moe":  # all experts chosen: rounding cannot flip a choice
        return replace(C.tiny_granite(hidden=1024, num_layers=2, num_heads=16, num_kv_heads=4, head_dim=64, ffn_dim=512),
                       num_experts=8, num_experts_per_tok=8), {PARTIAL, SWIGLU}
    return zozonex.model([zozonex.layer(zozonex.attn(heads=4, kv_heads=2, dim=64, vdim=64, window=60), 8200)] * 2, width=1024), {RELU2}


def _epilogues(run, *step, **kw):
    """The step's logits and the epilogues that the pair kernel ran with."""
    run.trace_begin(1 << 18)
    _, logits = run.run_flat(*step, want_logits=True, **kw)
    rec = run.trace_end(1 << 18)
    assert 0 < len(rec) < 1 << 18
    return logits, set(rec[rec[:, 1] == PAIR_KERNEL, 7].tolist())


@pytest.mark.parametrize("family", ["rms_swiglu_resid", "gelu", "relu2", "moe"])
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
        batch, ran = _epilogues(run, prompts, True, [0] * n, [[i] for i in range(n)], [0.0] * n)
        assert ran >= epilogues
        for i in range(n):
            one, ran = _epilogues(run, [prompts[i]], True, [0], [[i]], [0.0])
            assert not ran
            # the same bf16 roundings, sums in another order: an element may round the other way (2^-8 of it)
            rms = np.sqrt(np.mean((batch[i] - one[0]) ** 2) / np.mean(one[0] ** 2))
            assert rms <= 1e-2, f"sequence {i}: {rms}"
    finally:
        run.close()
