"""fp32 prompt attention with a tile's keys on one group of threads or shared by four (attention.cu): against the oracle around
the sizes where the rule changes sides, with a prompt that is found half cached."""
import pytest

from helpers import C, W, make_oracle, rel_err
import nvllm_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("head_dim", [16, 32, 64, 128])
@pytest.mark.parametrize("lens", [
    [9], [32],              # keys for two groups at most: one
    [33], [64, 65, 1],      # four; tiles that are full, of one key, of one query
    [200, 130],
    [70] * 24,              # more tiles than the chip holds CTAs: one
], ids=lambda n: f"{len(n)}x{n[0]}")
def test_prompts_match_the_oracle(head_dim, lens):
    cfg = C.tiny_llama(hidden=64, num_layers=2, num_heads=8, num_kv_heads=2, head_dim=head_dim, ffn_dim=64)
    prompts = [W.random_prompt(cfg.vocab_size, k, 70 + i).tolist() for i, k in enumerate(lens)]
    n = len(prompts)
    oracle = make_oracle(cfg, 4)
    exact = {i: oracle.greedy(prompts[i], 1)[1][0] for i in {0, n // 2, n - 1}}
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, W.random_weights(cfg, 4), precision=C.PREC_FP32, num_kv_blocks=n, sampling=None)
    try:
        for cached in (0, lens[0] // 2):
            logits = run.run_flat(prompts, True, [cached] + [0] * (n - 1), [[i] for i in range(n)], [0.0] * n, want_logits=True)[1]
            for i, want in exact.items():
                assert rel_err(logits[i], want) <= 1e-4  # what the fp32 mode is held to
    finally:
        run.close()
