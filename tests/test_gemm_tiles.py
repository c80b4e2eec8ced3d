"""The matrix kernels at the edges of their tiles, against float64 torch."""
import numpy as np
import pytest
import torch

from helpers import C, W, rel_err
import nvllm_pkg
import test_zozonex as zozonex

pytestmark = pytest.mark.gpu


def _product(M, N, K, prec, kernel):
    """Largest error over the bound of a K-term fp32 sum: K 2^-24 times the sum of the magnitudes of its terms."""
    L = nvllm_pkg.sub("lib")
    g = torch.Generator().manual_seed(M * 1000003 + N * 1009 + K)
    A, B = torch.randn(M, K, generator=g), torch.randn(K, N, generator=g)
    if prec == C.PREC_BF16:
        A, B = A.to(torch.bfloat16).float(), B.to(torch.bfloat16).float()
    out, _ = L.op_matmul(A.numpy(), B.numpy(), prec=prec, kernel=kernel)
    ref, mag = A.double() @ B.double(), A.double().abs() @ B.double().abs()
    return float(((torch.from_numpy(out).double() - ref).abs() / (mag * K * 2.0 ** -24 + 1e-30)).max())


@pytest.mark.parametrize("M,N,K", [
    (1, 1, 8), (9, 63, 24), (16, 64, 32), (17, 65, 40),  # 16- and 32-row tiles, columns around one tile, k tails
    (32, 130, 256), (33, 64, 264), (64, 192, 1000),      # the first 64-row tile, two and more k ranges
    (65, 3000, 136), (300, 768, 3072),                   # many tiles in one range; slices up to the buffer's room
])
def test_fp32_tiles(M, N, K):
    assert _product(M, N, K, C.PREC_FP32, 2) <= 1.0


@pytest.mark.parametrize("M,N,K", [
    (2, 1, 8), (3, 15, 72), (5, 17, 264), (8, 16, 64),   # rows, columns and k around one 16 x 64 chunk
    (7, 100, 776), (8, 768, 3072), (2, 2304, 768),       # k ranges on several CTAs
    (4, 9473, 520), (8, 9472, 4544),                     # the first column counts with 32-row tiles
])
def test_bf16_rows_on_mma(M, N, K):
    assert _product(M, N, K, C.PREC_BF16, 1) <= 1.0


@pytest.mark.parametrize("N,K", [(2048, 2048), (16384, 2048), (4672, 4544)])
def test_bf16_rows_on_mma_sum_as_exactly_as_single_rows(N, K):
    """The tensor core adds 16 products at a time; the error of the whole sum stays that of the CUDA-core kernel's chains of
    FMAs, which a single row takes (each side's 2-norm over some 10^4 outputs: known to a few percent)."""
    L = nvllm_pkg.sub("lib")
    g = torch.Generator().manual_seed(N + K)
    A, B = (torch.randn(*s, generator=g).to(torch.bfloat16).float() for s in ((4, K), (K, N)))
    ref = A.double() @ B.double()

    def error(rows):
        out = np.concatenate([L.op_matmul(A[r].numpy(), B.numpy(), prec=C.PREC_BF16, kernel=1)[0] for r in rows])
        return float((torch.from_numpy(out).double() - ref).norm())

    assert error([slice(0, 4)]) <= 1.1 * error([slice(i, i + 1) for i in range(4)])


@pytest.mark.parametrize("lens", [[600], [10] * 40])  # slices of the layers' products; of the head's
def test_fp32_step_does_not_depend_on_the_steps_before_it(lens):
    """How many k ranges the fp32 products take is decided by the step, not by the room that a larger step left behind."""
    R = nvllm_pkg.sub("runner")
    cfg = C.tiny_gpt2(hidden=512, num_heads=8, num_kv_heads=8, head_dim=64, ffn_dim=2048)
    run = R.CudaModelRunner(cfg, W.random_weights(cfg, 5), precision=C.PREC_FP32, num_kv_blocks=200, sampling=None)

    def step(lens):
        prompts = [W.random_prompt(cfg.vocab_size, k, 60 + i) for i, k in enumerate(lens)]
        return run.run_flat(prompts, True, [0] * len(lens), [[5 * i, 5 * i + 1, 5 * i + 2] if k > 256 else [i] for i, k in enumerate(lens)],
                            [0.0] * len(lens), want_logits=True)[1]

    try:
        first = step(lens)
        step([20] * 200)
        assert np.array_equal(step(lens), first)
    finally:
        run.close()


def test_fp32_rows_may_use_the_room_of_an_earlier_step():
    """Eight decoding sequences of a wide feed-forward: 72 slices of the second product, more than a workspace of eight rows
    has room for, but the prompts' has."""
    R = nvllm_pkg.sub("runner")
    cfg = C.tiny_gpt2(hidden=64, num_heads=4, num_kv_heads=4, head_dim=16, ffn_dim=36864)
    run = R.CudaModelRunner(cfg, W.random_weights(cfg, 5), precision=C.PREC_FP32, num_kv_blocks=8, sampling=None)
    prompts = [W.random_prompt(cfg.vocab_size, 90, 60 + i) for i in range(8)]
    tables, zeros = [[i] for i in range(8)], [0.0] * 8
    try:
        toks, _ = run.run_flat(prompts, True, [0] * 8, tables, zeros)
        texts = [np.append(p, t) for p, t in zip(prompts, toks)]
        _, eight = run.run_flat(texts, False, None, tables, zeros, want_logits=True)
        for i in range(8):
            _, one = run.run_flat([texts[i]], False, None, [tables[i]], [0.0], want_logits=True)
            assert rel_err(eight[i], one[0]) <= 1e-4
    finally:
        run.close()


@pytest.mark.parametrize("H", [8, 72, 1024, 2048, 2056, 4544, 8192])
@pytest.mark.parametrize("layer_norm", [False, True])
def test_norm_of_many_rows(H, layer_norm):
    """512 rows take the kernel that keeps a row in registers (one to four vectors per thread)."""
    L = nvllm_pkg.sub("lib")
    g = torch.Generator().manual_seed(H)
    x, w, b = torch.randn(512, H, generator=g) * 3 + 1, torch.randn(H, generator=g), torch.randn(H, generator=g)
    y, _ = L.op_norm(x.numpy(), w.numpy(), b.numpy() if layer_norm else None, eps=1e-5)
    xd = x.double() - (x.double().mean(-1, keepdim=True) if layer_norm else 0.0)
    ref = xd / torch.sqrt(xd.square().mean(-1, keepdim=True) + 1e-5) * w.double() + (b.double() if layer_norm else 0.0)
    # a few fp32 roundings of numbers up to ~10 times a weight, and a sum of H terms: 2^-24 (H / 256 + 16) of the largest
    assert float((torch.from_numpy(y).double() - ref).abs().max()) <= 2.0 ** -24 * (H / 256 + 16) * float(ref.abs().max())


NORM_ROWS_KERNEL = 47  # its id in the timeline; a record's last word says what the row took in before its norm
ADDEND, EXPERT_ROWS, SECOND_ADDEND, ON_THE_ADDEND = 1, 2, 4, 8


@pytest.mark.parametrize("family", ["llama", "falcon", "moe", "zozonex"])
def test_norm_of_many_rows_with_addends(family):
    """One pending product, two of them and a LayerNorm, the expert rows of a combine, a norm on the addend: float32 prompts
    as one batch, whose norms take the kernel for many rows, against the same prompts one at a time."""
    R = nvllm_pkg.sub("runner")
    if family == "zozonex":
        cfg, w = zozonex.random_weights(zozonex.model([zozonex.layer(zozonex.attn(), 96)] * 2, width=264), 3)
        weights, form = w.items(), ON_THE_ADDEND | ADDEND
    else:
        cfg, form = {"llama": (C.tiny_llama(hidden=264), ADDEND), "falcon": (C.tiny_falcon(), ADDEND | SECOND_ADDEND),
                     "moe": (C.tiny_granite(hidden=264), ADDEND | EXPERT_ROWS)}[family]
        weights = W.random_weights(cfg, 3)
    n = 24
    prompts = [W.random_prompt(cfg.vocab_size, 80 + (7 * i) % 23, 60 + i) for i in range(n)]  # 2199 rows: products in one slice
    run = R.CudaModelRunner(cfg, weights, precision=C.PREC_FP32, num_kv_blocks=n, sampling=None)

    def step(which):
        run.trace_begin(1 << 18)
        _, logits = run.run_flat([prompts[i] for i in which], True, [0] * len(which), [[i] for i in which], [0.0] * len(which),
                                 want_logits=True)
        rec = run.trace_end(1 << 18)
        assert 0 < len(rec) < 1 << 18
        return logits, set(rec[rec[:, 1] == NORM_ROWS_KERNEL, 7].tolist())

    try:
        batch, forms = step(range(n))
        assert form in forms
        for i in range(n):
            one, forms = step([i])
            assert not forms
            assert rel_err(batch[i], one[0]) <= 1e-4  # what the fp32 mode is held to against the reference
    finally:
        run.close()
