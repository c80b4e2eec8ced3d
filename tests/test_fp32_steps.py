"""fp32 steps of few rows: how the products' CTAs share the SMs, from the device timeline."""
import numpy as np
import pytest

from helpers import C, W
import nvllm_pkg

pytestmark = pytest.mark.gpu

GEMV, PRODUCT = 11, 12  # ids in the timeline


def timeline(cfg, n):
    """Records of a decode step of n sequences: sequence of the launch, kernel, CTA, SM, entry, after the wait, exit."""
    texts = [W.random_prompt(cfg.vocab_size, 6, i) for i in range(n)]
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, W.random_weights(cfg, 3), precision=C.PREC_FP32, num_kv_blocks=n, sampling=None)
    try:
        run.set_graphs(False)
        run.set_speculation(False)
        for _ in range(2):
            run.trace_begin(1 << 18)
            run.run_flat(texts, False, None, [[i] for i in range(n)], [0.0] * n)
            rec = run.trace_end(1 << 18).astype(np.int64)
        return [rec[rec[:, 0] == s] for s in np.unique(rec[:, 0])]
    finally:
        run.close()


def most_on_one_sm(rec):
    most = 0
    for sm in np.unique(rec[:, 3]):
        r = rec[rec[:, 3] == sm]
        most = max(most, max(int(((r[:, 4] <= t) & (r[:, 6] > t)).sum()) for t in r[:, 4]))
    return most


@pytest.mark.parametrize("n,ctas", [(1, 4), (2, 4), (3, 2), (4, 2), (5, 2), (6, 2)])
def test_ctas_of_a_product_on_an_sm(n, ctas):
    """256 threads with at most 64 registers (two weight rows to a warp), or 128 (four)."""
    cfg = C.tiny_llama(hidden=1024, ffn_dim=16384, num_layers=1)
    launches = [r for r in timeline(cfg, n) if r[0, 1] == GEMV]
    assert most_on_one_sm(max(launches, key=len)) >= ctas


@pytest.mark.parametrize("n", [9, 16])
def test_the_kernel_behind_a_product_comes_late(n):
    """CTAs that come in while a product's own still fill the SMs unevenly stay where they are (gemm_simt.cu)."""
    launches = timeline(C.tiny_llama(hidden=1024, ffn_dim=16384, num_layers=1), n)
    seen = 0
    for rec, behind in zip(launches, launches[1:]):
        if rec[0, 1] == PRODUCT and len(rec) >= 100:
            start, end = rec[:, 4].max(), rec[:, 6].max()
            assert behind[:, 4].min() >= start + (end - start) // 3
            seen += 1
    assert seen >= 2
