"""Steps of one bf16 row (gemv_row.cu: norm in front of a product, activation or residual update behind it) against the same
sequences decoded as one batch, whose products, norms and activations are other kernels."""
import numpy as np
import pytest

from helpers import C, W
import nvllm_pkg

pytestmark = pytest.mark.gpu

KERNEL = 50  # its id in the timeline


def gpt2(hidden, ffn, heads=2):
    return C.tiny_gpt2(hidden=hidden, num_layers=2, num_heads=heads, num_kv_heads=heads, head_dim=64, ffn_dim=ffn)


def llama(hidden, ffn):
    return C.tiny_llama(hidden=hidden, num_layers=2, num_heads=4, num_kv_heads=2, head_dim=64, ffn_dim=ffn)


@pytest.mark.parametrize("cfg", [
    gpt2(128, 72),                             # one piece a lane; part of one
    gpt2(264, 768, heads=3), gpt2(768, 776),   # three pieces; into the fourth
    gpt2(1024, 1032), llama(1032, 2048),       # one warp a row; two, the last piece empty
    llama(2056, 4096), llama(4096, 8192),      # four; eight
    llama(520, 8200),                          # feed-forward wider than this kernel takes: the first layer's projections alone
    llama(4104, 512),                          # rows wider than it norms
], ids=lambda c: f"{c.hidden}-{c.ffn_dim}")
def test_one_row_matches_the_batch(cfg):
    n, steps = 9, 2
    prompts = [W.random_prompt(cfg.vocab_size, 5 + 3 * i, 60 + i) for i in range(n)]
    more = [W.random_prompt(cfg.vocab_size, steps, 90 + i) for i in range(n)]
    weights = list(W.random_weights(cfg, 7, round_bf16=True))

    def logits(precision, which, trace=False):
        """The steps' logits of the sequences in `which`, all in one batch."""
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, weights, precision=precision, num_kv_blocks=n, sampling=None)
        try:
            run.set_graphs(False)
            if trace:
                run.trace_begin(1 << 18)
            run.run_flat([prompts[i] for i in which], True, [0] * len(which), [[i] for i in which], [0.0] * len(which))
            out = [run.run_flat([np.concatenate([prompts[i], more[i][:k + 1]]) for i in which], False, None,
                                [[i] for i in which], [0.0] * len(which), want_logits=True)[1] for k in range(steps)]
            return (np.stack(out), KERNEL in run.trace_end(1 << 18)[:, 1]) if trace else np.stack(out)
        finally:
            run.close()

    want, batch = logits(C.PREC_FP32, range(n)), logits(C.PREC_BF16, range(n))
    rows = [logits(C.PREC_BF16, [i], trace=True) for i in range(n)]
    assert all(ran == (cfg.hidden <= 4096) for _, ran in rows)
    alone = np.concatenate([out for out, _ in rows], 1)
    # the same bf16 roundings, sums in another order: as far from float32 as the batch is (the error's norm over n sequences
    # of one step is known to a tenth or so)
    assert np.linalg.norm(alone - want) <= 1.25 * np.linalg.norm(batch - want)
