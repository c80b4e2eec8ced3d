"""Windows of keys in the tcgen05 prompt attention (attention_tc5.cu): bf16 prompts against the fp32 mode, whose attention is
another kernel, with windows around the edges of its key tiles and chunks and prompts cut into portions."""
import numpy as np
import pytest

from helpers import C, W
import nvllm_pkg
import test_zozonex as zozonex

pytestmark = pytest.mark.gpu

KERNEL = 13  # its id in the timeline


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("window", [1, 32, 33, 63, 64, 65, 127, 128, 129, 300, 2000])
def test_prompts_match_the_fp32_mode(dim, window):
    mix = zozonex.attn(heads=3, kv_heads=1, dim=dim, vdim=dim, window=window)
    cfg, w = zozonex.random_weights(zozonex.model([zozonex.layer(mix, 96)] * 2, width=128), 5, bf16=True)
    lens, first = [385, 1, 130, 257], [200, 0, 128, 0]  # tokens; of them computed in an earlier step
    texts = [W.random_prompt(cfg.vocab_size, k, 60 + i) for i, k in enumerate(lens)]
    tables = [[4, 2], [0], [1], [5, 3]]

    def logits(precision):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, w.items(), precision=precision, num_kv_blocks=6, sampling=None)
        try:
            run.trace_begin(1 << 18)
            early = [i for i, k in enumerate(first) if k]
            run.run_flat([texts[i][:first[i]] for i in early], True, [0] * len(early), [tables[i] for i in early], [0.0] * len(early))
            out = run.run_flat(texts, True, first, tables, [0.0] * len(texts), want_logits=True)[1]
            return out, KERNEL in run.trace_end(1 << 18)[:, 1]
        finally:
            run.close()

    want, ran = logits(C.PREC_FP32)
    assert not ran
    got, ran = logits(C.PREC_BF16)
    assert ran
    # two layers of bf16 roundings (2^-9 an operand, some ten of them in a row); a key too many or too few shows as 1 / window
    rms = np.sqrt(((got - want) ** 2).mean(1) / (want ** 2).mean(1))
    assert (rms <= 2e-2).all(), rms
