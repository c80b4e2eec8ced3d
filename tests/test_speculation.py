"""The speculative next step of nvllm_run: calls that never ask for it pause it, a decode loop gets it back, and results (tokens,
logits, device time of the step that was asked for) are those of a runner without it."""
import numpy as np
import pytest

from helpers import C, W
import nvllm_pkg

pytestmark = pytest.mark.gpu


def test_prompts_pause_it_and_decoding_brings_it_back():
    cfg = C.tiny_llama()
    prompts = [W.random_prompt(cfg.vocab_size, 18 + 7 * i, 300 + i).tolist() for i in range(3)]
    tables = [[i] for i in range(3)]

    def drive(spec):
        run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, W.random_weights(cfg, 5), precision=C.PREC_FP32, num_kv_blocks=3, sampling=None)
        try:
            run.set_speculation(spec)
            outs, hits = [], []
            for _ in range(12):  # each call after a speculation is a miss; the pauses grow to 16 calls
                outs.append(run.run_flat(prompts, True, [0] * 3, tables, [0.0] * 3, want_logits=True))
            seqs = [list(p) for p in prompts]
            for k in range(40):
                for s, t in zip(seqs, outs[-1][0]):
                    s.append(int(t))
                outs.append(run.run_flat(seqs, False, None, tables, [0.0] * 3, want_logits=k % 2 == 0))
                hits.append(run.last_stats.h2d_bytes == 0)
                assert run.last_stats.device_ms > 0
            return outs, hits
        finally:
            run.close()

    (want, none), (got, hits) = drive(False), drive(True)
    assert not any(none)
    first = hits.index(True)
    assert first <= 17 and all(hits[first:])
    for (a, la), (b, lb) in zip(want, got):
        np.testing.assert_array_equal(a, b)
        assert (la is None) == (lb is None)
        if la is not None:
            np.testing.assert_array_equal(la, lb)  # same kernels, same order
