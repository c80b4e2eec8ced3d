"""A bounded wait inside a kernel that runs out is reported to the caller whose launch it was, and to nobody else.  The
failure is made on the host (nvllm_inject_wait_failure does there what the kernel does); no wait runs out on the device."""
import os
import re
import threading

import numpy as np
import pytest

from helpers import C, ROOT, W
import nvllm_pkg

gpu = pytest.mark.gpu


def _runner(seed):
    R = nvllm_pkg.sub("runner")
    cfg = C.tiny_llama()
    return R.CudaModelRunner(cfg, W.random_weights(cfg, seed, round_bf16=True), precision=C.PREC_BF16, num_kv_blocks=4, sampling=None)


def test_limits_count_from_the_launch_dependency():
    """Under programmatic launch a CTA may start long before the kernels in front are done: each role of the pair kernel
    waits for them, in dense and grouped products alike, before its first wait with a limit."""
    with open(os.path.join(ROOT, "nano-vllm-go_b200", "csrc", "gemm_tc5_pair.cu")) as f:
        kernel = f.read().split("\ngemm_tc5_pair_kernel(", 1)[1].split("\n}\n", 1)[0]
    roles = re.split(r"\n  (?:if \(warp == 0\) \{\n    uint64_t|\} else if \(warp == 1\) \{|\} else \{)", kernel)[1:]
    assert len(roles) == 3
    for role in roles:
        dependency = re.search(r"^ +pdl_wait\(\);", role, re.M)
        assert dependency and dependency.start() < role.index("wait_limited(")


@gpu
def test_only_the_handle_whose_wait_ran_out_fails():
    L = nvllm_pkg.sub("lib")
    a, b = _runner(1), _runner(2)
    prompt = [int(t) for t in W.random_prompt(a.cfg.vocab_size, 20, 3)]
    try:
        want = {r: r.run_flat([prompt], True, [0], [[0]], [0.0], want_logits=True)[1] for r in (a, b)}
        L.check(L.load().nvllm_inject_wait_failure(a._h), a._h)
        for _ in range(2):  # b synchronises first, in both of the calls that hand out results
            assert np.array_equal(b.run_flat([prompt], True, [0], [[0]], [0.0], want_logits=True)[1], want[b])
            b.sync()
        with pytest.raises(L.NvllmError, match="wait") as err:
            a.run_flat([prompt], True, [0], [[0]], [0.0])
        assert err.value.code == L.ERR_CUDA
        # nothing goes on from the step that failed
        for call in (a.run_resident, a.rerun):
            with pytest.raises(L.NvllmError) as err:
                call()
            assert err.value.code == L.ERR_STATE
        # and the next step is an ordinary one
        assert np.array_equal(a.run_flat([prompt], True, [0], [[0]], [0.0], want_logits=True)[1], want[a])
        L.check(L.load().nvllm_inject_wait_failure(a._h), a._h)
        with pytest.raises(L.NvllmError, match="wait"):
            a.sync(1)
        with pytest.raises(L.NvllmError) as err:
            a.run_resident()
        assert err.value.code == L.ERR_STATE
    finally:
        a.close()
        b.close()


@gpu
def test_a_matrix_product_whose_wait_ran_out_fails_and_no_later_call():
    L = nvllm_pkg.sub("lib")
    x, w = np.ones((300, 64), np.float32), np.ones((64, 512), np.float32)
    L.check(L.load().nvllm_inject_wait_failure(None))
    other = []
    t = threading.Thread(target=lambda: other.append(L.op_matmul(x, w, prec=C.PREC_BF16, kernel=3)[0]))
    t.start()
    t.join()
    assert other and np.all(other[0] == 64.0)
    with pytest.raises(L.NvllmError, match="wait") as err:
        L.op_matmul(x, w, prec=C.PREC_BF16, kernel=3)
    assert err.value.code == L.ERR_CUDA
    assert np.all(L.op_matmul(x, w, prec=C.PREC_BF16, kernel=3)[0] == 64.0)
    run = _runner(1)
    try:
        run.run_flat([[1, 2, 3]], True, [0], [[0]], [0.0])
    finally:
        run.close()
