"""Granite-4 hybrid (Mamba2 + attention blocks): the CUDA path against the
oracle's restatement of purego/tensor/mamba2.go (itself pinned to an independent numpy
restatement in tests/test_oracle.py).  Ragged batches, decode steps that carry the SSM state
through the per-KV-block snapshots, a sequence crossing a 256-token block boundary."""
import numpy as np
import pytest

from helpers import C, W, make_oracle, oracle_mod, rel_err
import nvllm_pkg

pytestmark = pytest.mark.gpu
TOL = {C.PREC_FP32: 1e-4, C.PREC_BF16: 2e-2}


def _run(cfg, prec, prompts, steps, tables, num_kv_blocks, **kw):
    R = nvllm_pkg.sub("runner")
    bf16 = prec == C.PREC_BF16
    orc = make_oracle(cfg, round_bf16=bf16)
    refs = [orc.greedy(p, steps) for p in prompts]
    run = R.CudaModelRunner(cfg, W.random_weights(cfg, 1234, round_bf16=bf16), precision=prec,
                            num_kv_blocks=num_kv_blocks, sampling=None, **kw)
    worst, flips = 0.0, 0
    try:
        seqs = [[int(t) for t in p] for p in prompts]
        n = len(seqs)
        for i in range(steps):
            out, logits = run.run_flat(seqs, i == 0, [0] * n if i == 0 else None, tables, [0.0] * n,
                                       want_logits=True)
            for s in range(n):
                ref = refs[s][1][i]
                err = rel_err(logits[s], ref)
                worst = max(worst, err)
                assert err <= TOL[prec], f"seq {s} step {i}: rel err {err}"
                assert int(out[s]) == oracle_mod().argmax(logits[s])
                if int(out[s]) != int(refs[s][0][i]):
                    margin = float(ref[refs[s][0][i]] - ref[out[s]])
                    assert bf16 and margin <= 2 * err * float(np.abs(ref).max()) + 1e-6
                    flips += 1
                seqs[s].append(int(refs[s][0][i]))
        assert flips <= 1
    finally:
        run.close()
    return worst


@pytest.mark.parametrize("prec", [C.PREC_FP32, C.PREC_BF16])
def test_hybrid_single_sequence(prec):
    cfg = C.tiny_hybrid()
    _run(cfg, prec, [W.random_prompt(cfg.vocab_size, 40, 1)], 6, [[0]], 2)


@pytest.mark.parametrize("prec", [C.PREC_FP32, C.PREC_BF16])
def test_hybrid_ragged_batch_crossing_a_block_boundary(prec):
    """Three sequences; the 250-token one reaches position 256 during the decode steps, so its SSM
    state moves from block to block through the snapshots."""
    cfg = C.tiny_hybrid()
    prompts = [W.random_prompt(cfg.vocab_size, n, 10 + i) for i, n in enumerate((250, 17, 300))]
    _run(cfg, prec, prompts, 10, [[0, 1], [2], [3, 4]], 6)


def test_hybrid_larger_state_and_groups():
    """state 64 / head_dim 64 / 1 group / 3 conv taps, batch of 12 decode rows (tcgen05 GEMM tiles)."""
    cfg = C.tiny_hybrid(mamba_num_heads=4, mamba_head_dim=64, mamba_state_size=64, mamba_n_groups=1,
                        mamba_conv_kernel=3, hybrid_layers=(True, True, False, True))
    prompts = [W.random_prompt(cfg.vocab_size, 20 + i, 30 + i) for i in range(12)]
    _run(cfg, C.PREC_BF16, prompts, 4, [[i] for i in range(12)], 12, max_num_seqs=16)


def test_hybrid_resident_decode_matches_stepwise():
    """nvllm_run_resident (device-side advance, CUDA graph) on a hybrid model."""
    R = nvllm_pkg.sub("runner")
    cfg = C.tiny_hybrid()
    prompt = [int(t) for t in W.random_prompt(cfg.vocab_size, 30, 3)]
    outs = []
    for resident in (False, True):
        run = R.CudaModelRunner(cfg, W.random_weights(cfg, 1234), precision=C.PREC_FP32, num_kv_blocks=2,
                                sampling=None)
        toks = list(prompt)
        o, _ = run.run_flat([toks], True, [0], [[0]], [0.0])
        toks.append(int(o[0]))
        o, _ = run.run_flat([toks], False, None, [[0]], [0.0])
        toks.append(int(o[0]))
        for _ in range(12):
            if resident:
                run.run_resident()
                o, _ms = run.sync(1)
            else:
                o, _ = run.run_flat([toks], False, None, [[0]], [0.0])
            toks.append(int(o[0]))
        run.close()
        outs.append(toks)
    assert outs[0] == outs[1]


def test_hybrid_rejects_multi_token_prefill_on_a_cached_prefix():
    R = nvllm_pkg.sub("runner")
    L = nvllm_pkg.sub("lib")
    cfg = C.tiny_hybrid()
    run = R.CudaModelRunner(cfg, W.random_weights(cfg, 1234), precision=C.PREC_FP32, num_kv_blocks=4,
                            sampling=None)
    try:
        p = [int(t) for t in W.random_prompt(cfg.vocab_size, 300, 2)]
        run.run_flat([p], True, [0], [[0, 1]], [0.0])
        with pytest.raises(L.NvllmError, match="Mamba2"):
            run.run_flat([p], True, [256], [[0, 1]], [0.0])
        run.run_flat([p + [5]], True, [300], [[0, 1]], [0.0])  # decode-shaped: fine
    finally:
        run.close()


@pytest.mark.parametrize("nh,hd,N,G,K", [
    (8, 4, 16, 1, 4),     # smallest head of the tiled scan: two heads to a warp and more
    (8, 64, 64, 2, 4),
    (4, 128, 128, 4, 4),  # largest head and state, one head per group
    (32, 128, 16, 8, 4),  # eight sequences of that many heads are enough warps for twice the rows per lane
    (32, 128, 32, 8, 4),
    (32, 128, 64, 8, 4),
    (32, 128, 128, 8, 4),
    (8, 32, 24, 2, 4),    # state that is no power of two: the scan without tiles
    (6, 12, 16, 3, 4),    # rows that start off 16-byte boundaries
    (8, 32, 16, 2, 3),    # other taps
])
def test_hybrid_prompts_at_the_edges_of_the_scan_tiles(nh, hd, N, G, K):
    """Prompts of one token, around the scan's chunk of sixteen and over a block border, decoded on."""
    cfg = C.tiny_hybrid(vocab_size=256, num_layers=2, hybrid_layers=(True, True), mamba_num_heads=nh, mamba_head_dim=hd,
                        mamba_state_size=N, mamba_n_groups=G, mamba_conv_kernel=K)
    prompts = [W.random_prompt(cfg.vocab_size, n, 50 + i) for i, n in enumerate((1, 7, 15, 16, 17, 32, 33, 258))]
    _run(cfg, C.PREC_FP32, prompts, 3, [[i] for i in range(7)] + [[7, 8]], 9)


def test_hybrid_scan_with_sixteen_heads_to_a_cta():
    """The smallest heads, one group, and so many short prompts that a lane holds two rows of a head: 16 heads per CTA.
    (771 rows: also enough for the convolution's windows, with several sequences in each.)"""
    cfg = C.tiny_hybrid(vocab_size=256, num_layers=2, hybrid_layers=(True, True), mamba_num_heads=64, mamba_head_dim=4,
                        mamba_state_size=16, mamba_n_groups=1, mamba_conv_kernel=4)
    prompts = [W.random_prompt(cfg.vocab_size, 1 + i % 21, 50 + i) for i in range(75)]
    _run(cfg, C.PREC_FP32, prompts, 3, [[i] for i in range(75)], 75)


@pytest.mark.parametrize("N,hd,n", [(16, 8, 1), (32, 32, 1), (64, 16, 1), (128, 64, 1), (128, 128, 20)])  # (the last: 1280 warps)
def test_hybrid_decays_of_every_strength(N, hd, n):
    """The tiled scan keeps the state divided by the product of its decays: heads whose decays are near one, small
    enough that the product leaves fp32's range inside a chunk of tokens, and zero."""
    R = nvllm_pkg.sub("runner")
    cfg = C.tiny_hybrid(vocab_size=256, num_layers=2, hybrid_layers=(True, True), mamba_num_heads=8, mamba_head_dim=hd,
                        mamba_state_size=N, mamba_n_groups=2, mamba_conv_kernel=4)
    a_log = np.array([-6.0, 0.0, 1.0, 2.0, 3.0, 4.5, 6.0, -1.0], dtype=np.float32)

    def weights():
        for wid, layer, w in W.random_weights(cfg, 1234):
            yield wid, layer, a_log if wid == C.W_MAMBA_A_LOG else w

    prompt = [int(t) for t in W.random_prompt(cfg.vocab_size, 70, 9)]
    ref = oracle_mod().OracleModel(cfg, weights())
    want = ref.greedy(prompt, 2)
    run = R.CudaModelRunner(cfg, weights(), precision=C.PREC_FP32, num_kv_blocks=n, sampling=None)
    tables, zeros = [[i] for i in range(n)], [0] * n
    try:
        _, logits = run.run_flat([prompt] * n, True, zeros, tables, zeros, want_logits=True)
        assert max(rel_err(row, want[1][0]) for row in logits) <= 1e-4
        _, logits = run.run_flat([prompt + [int(want[0][0])]] * n, False, None, tables, zeros, want_logits=True)
        assert max(rel_err(row, want[1][1]) for row in logits) <= 1e-4
    finally:
        run.close()


CONV, SCAN = 20, 21  # ids in the timeline


def test_hybrid_decode_scan_grows_with_the_batch_only():
    """A decode step's scan is bound by the state that it reads and writes: four times the sequences, four times the time."""
    cfg = C.tiny_hybrid(vocab_size=256, num_layers=1, hybrid_layers=(True,), mamba_num_heads=64, mamba_head_dim=64,
                        mamba_state_size=128, mamba_n_groups=1, mamba_conv_kernel=4)
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, W.random_weights(cfg, 7), precision=C.PREC_BF16, num_kv_blocks=512, sampling=None)
    times = {}
    try:
        for n in (128, 512):
            seqs, tables = [[i % 256, 3] for i in range(n)], [[i] for i in range(n)]
            for _ in range(3):
                run.trace_begin(1 << 17)
                run.run_flat(seqs, False, None, tables, [0.0] * n)
                rec = run.trace_end(1 << 17)
                took = int(rec[rec[:, 1] == SCAN, 6].max()) - int(rec[rec[:, 1] == CONV, 6].max())
                times[n] = min(times.get(n, took), took)
    finally:
        run.close()
    assert times[512] <= 6 * times[128], times  # (four, and half as much again for what a small batch hides)


@pytest.mark.parametrize("lengths", [
    (9, 9, 9), (3, 40, 3), tuple(1 + i % 2 for i in range(7)),                         # all alike; one of them longer; ties
    tuple(5 + 37 * i % 61 for i in range(64)), tuple(1 + 7 * i % 19 for i in range(520)),  # in no order; more than 512 of them
], ids=lambda v: str(len(v)))
def test_hybrid_prompts_of_any_lengths_are_what_each_is_alone(lengths):
    """The scan takes the sequences of a step by length (mamba.cu): each ends as it does alone, now and in a step that is repeated."""
    cfg = C.tiny_hybrid(vocab_size=256, num_layers=2, hybrid_layers=(True, True), mamba_num_heads=4, mamba_head_dim=16,
                        mamba_state_size=32, mamba_n_groups=1, mamba_conv_kernel=4)
    n = len(lengths)
    seqs = [W.random_prompt(cfg.vocab_size, k, 50 + i).tolist() for i, k in enumerate(lengths)]
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, W.random_weights(cfg, 7), precision=C.PREC_FP32, num_kv_blocks=n + 1, sampling=None)
    try:
        out, logits = run.run_flat(seqs, True, [0] * n, [[i] for i in range(n)], [0.0] * n, want_logits=True)
        after = run.run_flat([s + [int(t)] for s, t in zip(seqs, out)], False, None, [[i] for i in range(n)], [0.0] * n, want_logits=True)
        for i in sorted({0, 1, n // 2, n - 1, int(np.argmax(lengths)), int(np.argmin(lengths))}):
            one, alone = run.run_flat([seqs[i]], True, [0], [[n]], [0.0], want_logits=True)
            assert rel_err(logits[i], alone[0]) <= TOL[C.PREC_FP32] and int(one[0]) == int(out[i])
            _, alone = run.run_flat([seqs[i] + [int(out[i])]], False, None, [[n]], [0.0], want_logits=True)
            assert rel_err(after[1][i], alone[0]) <= TOL[C.PREC_FP32]
        run.run_flat(seqs, True, [0] * n, [[i] for i in range(n)], [0.0] * n)
        run.rerun()
        np.testing.assert_array_equal(run.sync(n)[0], out)
    finally:
        run.close()
