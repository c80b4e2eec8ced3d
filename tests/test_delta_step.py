"""Decode steps of the delta rule (delta_step_kernel): tokens one at a time against the same texts as prompts, whose
convolution and scan are other kernels, and against the float64 restatement, in the fp32 mode."""
import numpy as np
import pytest

from helpers import C, W, rel_err
import nvllm_pkg
import test_zozonex as zozonex

pytestmark = pytest.mark.gpu

KERNEL = 51  # its id in the timeline


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,conv,taken", [
    (4, 2, 128, 128, 4, True),   # two heads share q and k: their tails move on behind the kernel
    (2, 2, 64, 64, 2, True),     # one block of columns, one older row in the tail
    (4, 1, 128, 64, 3, True),
    (3, 1, 128, 64, 3, False),   # gates off the 16-byte boundaries
    (2, 1, 64, 128, 4, True),
    (2, 1, 64, 96, 4, False),    # columns that don't fill its blocks
    (2, 1, 64, 64, 1, False),    # no tail
])
def test_tokens_one_at_a_time_match_prompts(heads, kv_heads, dim, vdim, conv, taken):
    model = zozonex.model([zozonex.layer(zozonex.delta(heads, kv_heads, dim, vdim, conv), 96)] * 2, width=128)
    cfg, w = zozonex.random_weights(model, 5)
    n, steps = 3, 7
    texts = [W.random_prompt(cfg.vocab_size, 1 + i * i + steps, 60 + i) for i in range(n)]  # starts of 1, 2 and 5 tokens
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, w.items(), precision=C.PREC_FP32, num_kv_blocks=n, sampling=None, num_state_slots=n)
    slots = [2, 0, 1]

    def step(lens, prefill, which=range(n)):
        return run.run_flat([texts[i][:k] for i, k in zip(which, lens)], prefill, [0] * len(lens) if prefill else None,
                            [[i] for i in which], [0.0] * len(lens), want_logits=True, state_slots=[slots[i] for i in which])[1]

    try:
        run.set_graphs(False)
        run.trace_begin(1 << 18)
        lens = np.array([len(t) - steps for t in texts])
        got = [step(lens, True)]
        for _ in range(steps):
            lens += 1
            got.append(step(lens, False))
        got.append(step([1] * n, True))  # one-token prompts: whatever the slots hold counts as nothing
        got.append(step([2] * n, False))
        assert (KERNEL in run.trace_end(1 << 18)[:, 1]) == taken
        for i in range(n):
            exact = zozonex.ref.forward(model, w, texts[i])
            for k in range(steps + 1):
                assert rel_err(got[k][i], exact[len(texts[i]) - steps + k - 1]) <= 1e-4, (k, i)  # what the fp32 mode is held to
        for k in range(steps + 1):
            for i in range(n):
                want = step([len(texts[i]) - steps + k], True, [i])[0]
                assert rel_err(got[k][i], want) <= 1e-5, (k, i)  # 32-bit sums of some hundred terms in another order, two layers
        for k in (1, 2):
            for i in range(n):
                assert rel_err(got[steps + k][i], step([k], True, [i])[0]) <= 1e-5, (k, i)
    finally:
        run.close()
