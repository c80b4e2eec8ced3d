"""Embedding rows of prompts (elementwise.cu launch_embed): a block or a warp per row, by how many there are; each prompt ends as it
does alone."""
import numpy as np
import pytest

from helpers import C, W, rel_err
import nvllm_pkg
import test_zozonex as zozonex

pytestmark = pytest.mark.gpu

EMBED = 5  # id in the timeline


def uniform(make, **kw):
    cfg = make(num_layers=1, **kw)
    return cfg, list(W.random_weights(cfg, 3))


def sines():
    cfg, w = zozonex.random_weights(zozonex.model([zozonex.layer(zozonex.attn(heads=2, kv_heads=1, dim=16, vdim=16, window=40))]), 7)
    return cfg, list(w.items())


@pytest.mark.parametrize("make,rows,warps", [
    (lambda: uniform(C.tiny_gpt2), 1775, False), (lambda: uniform(C.tiny_gpt2), 1776, True),
    (lambda: uniform(C.tiny_llama, hidden=1032), 1779, True),  # rows beside the last full CTA; a part of a warp's piece
    (lambda: uniform(C.tiny_granite), 512, False),
    (sines, 1776, False), (sines, 9471, False), (sines, 9472, True),
], ids=lambda v: str(v) if not callable(v) else "m")
def test_prompts_are_what_each_is_alone(make, rows, warps):
    cfg, weights = make()
    lengths = [50] * (rows // 50) + ([rows % 50] if rows % 50 else [])
    n = len(lengths)
    texts = [W.random_prompt(cfg.vocab_size, k, 160 + i) for i, k in enumerate(lengths)]
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, weights, precision=C.PREC_FP32, num_kv_blocks=n, sampling=None)
    try:
        run.set_speculation(False)
        run.trace_begin(1 << 19)
        logits = run.run_flat(texts, True, [0] * n, [[i] for i in range(n)], [0.0] * n, want_logits=True)[1]
        ctas = int((run.trace_end(1 << 19)[:, 1] == EMBED).sum())
        assert ctas == (-(-rows // 8) if warps else rows)
        for i in (0, n // 2, n - 1):
            alone = run.run_flat([texts[i]], True, [0], [[i]], [0.0], want_logits=True)[1]
            assert rel_err(logits[i], alone[0]) <= 1e-4  # what the fp32 mode is held to against the reference
    finally:
        run.close()
