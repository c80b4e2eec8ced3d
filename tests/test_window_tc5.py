"""Windows of keys in the tcgen05 prompt attention (attention_tc5.cu): bf16 prompts against the float64 restatement, with windows
around the edges of its key tiles and chunks, prompts cut into portions, and more items than the chip holds CTAs."""
import numpy as np
import pytest

from helpers import C, W
import nvllm_pkg
import test_zozonex as zozonex

pytestmark = pytest.mark.gpu

KERNEL = 13  # its id in the timeline
TILE = 128   # queries of an item


def attention(q, k, v, scale, window):
    """zozonex_ref.window_attention with all rows at once."""
    back = np.arange(len(q))[:, None] - np.arange(len(q))[None, :]
    s = np.where((back >= 0) & (back < window), q @ k.T * scale, -np.inf)
    mx = np.maximum(s.max(1, keepdims=True), 0.0)
    e = np.exp(s - mx)
    return (e / (np.exp(-mx) + e.sum(1, keepdims=True))) @ v


def setup(dim, window, heads, lens):
    mix = zozonex.attn(heads=heads, kv_heads=heads // 3, dim=dim, vdim=dim, window=window)
    model = zozonex.model([zozonex.layer(mix)], width=128)
    cfg, w = zozonex.random_weights(model, 5, bf16=True)
    texts = [W.random_prompt(cfg.vocab_size, k, 60 + i) for i, k in enumerate(lens)]
    pages = np.random.RandomState(3).permutation(2 * len(lens))
    return model, cfg, w, texts, [pages[2 * i:2 * i + 2].tolist() for i in range(len(lens))]


def prompts(cfg, w, texts, tables, first):
    """The logits of all rows behind the first ones, which an earlier step computes; and whether the kernel ran."""
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, w.items(), precision=C.PREC_BF16, num_kv_blocks=2 * len(texts), sampling=None)
    try:
        run.trace_begin(1 << 18)
        early = [i for i, k in enumerate(first) if k]
        run.run_flat([texts[i][:first[i]] for i in early], True, [0] * len(early), [tables[i] for i in early], [0.0] * len(early))
        rows = sum(len(t) - k for t, k in zip(texts, first))
        run.request_logits(np.arange(rows))
        run.run_flat(texts, True, first, tables, [0.0] * len(texts))
        return run.fetch_logits(rows), KERNEL in run.trace_end(1 << 18)[:, 1]
    finally:
        run.close()


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("window", [1, 32, 33, 63, 64, 65, 127, 128, 129, 300, 2000])
def test_prompts_match_float64_with_this_window_and_no_other(monkeypatch, dim, window):
    heads = 12
    lens = [385, 1, 130, 257] + [300 + 17 * i % 90 for i in range(10)]
    first = [200, 0, 128, 0] + [37 * i % 100 for i in range(10)]
    assert heads * sum(-(-(k - f) // TILE) for k, f in zip(lens, first)) > 2 * 148
    model, cfg, w, texts, tables = setup(dim, window, heads, lens)
    got, ran = prompts(cfg, w, texts, tables, first)
    assert ran
    monkeypatch.setattr(zozonex.ref, "window_attention", attention)

    def want(size):
        model["layers"][0]["mixer"]["mask"]["size"] = size
        return np.concatenate([zozonex.ref.forward(model, w, t)[f:] for t, f in zip(texts, first)])

    exact = want(window)
    off = got - exact
    # one layer of bf16 roundings: 2^-9 an operand, some eight of them in a row
    rms = np.sqrt((off ** 2).mean(1) / (exact ** 2).mean(1))
    assert rms.max() <= 2e-2
    # the differences lean towards a window of one key more or less by no part of the way there: rounding errors point
    # anywhere, and over some hundred rows of 128 independent logits a sum of them three times as large as a key's
    # share leans by 3 / sqrt(rows) of it.  Each quarter of an item (a warp's rows) by itself.
    quarter = np.concatenate([np.arange(k - f) % TILE // 32 for k, f in zip(lens, first)])
    for other in {window - 1, window + 1} - {0}:
        lean = want(other) - exact
        for q in range(4):
            a, b = off[quarter == q], lean[quarter == q]
            if (b != 0).any():
                assert abs((a * b).sum()) <= 0.25 * (b * b).sum(), (other, q)


@pytest.mark.parametrize("dim", [64, 128])
def test_a_window_of_any_size_is_no_window(dim):
    """The largest size that a configuration holds: the masks' sums stay within 32 bits, also where a portion's first row
    stands before a key tile (portions that begin off a multiple of 32)."""
    lens, first = [385, 300, 130], [200, 77, 0]
    _, cfg, w, texts, tables = setup(dim, 0, 3, lens)
    want, ran = prompts(cfg, w, texts, tables, first)
    assert ran
    for window in (2 ** 31 - 1, 2 ** 31 - 20, 512):
        _, cfg, w, texts, tables = setup(dim, window, 3, lens)
        got, ran = prompts(cfg, w, texts, tables, first)
        assert ran
        np.testing.assert_array_equal(got, want)  # the same products, sums in the same order
