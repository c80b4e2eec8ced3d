"""The fp32 product on split operands (gemm_f32_tc5.cu): against float64 at the edges of its tiles and slices, and with
operands whose split is not finite."""
import numpy as np
import pytest
import torch

from helpers import C, W
import nvllm_pkg

L = nvllm_pkg.sub("lib")
pytestmark = pytest.mark.gpu

KERNEL = 49  # its id in the timeline


def _run(A, Wm):
    """The product and whether this kernel made it."""
    cfg = C.tiny_gpt2()
    run = nvllm_pkg.sub("runner").CudaModelRunner(cfg, W.random_weights(cfg, 1), num_kv_blocks=1, sampling=None)
    try:
        run.trace_begin(1 << 16)
        out, _ = L.op_matmul(A, Wm, prec=C.PREC_FP32, kernel=2)
        rec = run.trace_end(1 << 16)
    finally:
        run.close()
    return out, bool((rec[:, 1] == KERNEL).any())


def _operands(M, N, K):
    g = torch.Generator().manual_seed(M * 31 + N * 7 + K)
    return torch.randn(M, K, generator=g).numpy(), torch.randn(K, N, generator=g).numpy()


def _error(out, A, Wm):
    """Largest error over its bound: in units of 2^-24 times the sum of the magnitudes of an element's terms, two for each of
    the 24 tensor-core sums of a stage, one per stage for the fp32 sums, one per slice, and 2 for the parts left out."""
    a, w = torch.from_numpy(A).cuda().double(), torch.from_numpy(Wm).cuda().double()
    bound = 2.0 ** -24 * (48 + A.shape[1] / 64 + 8 + 2) * (a.abs() @ w.abs())
    return float(((torch.from_numpy(out).cuda().double() - a @ w).abs() / bound).max())


@pytest.mark.parametrize("M,N,K,tc", [
    (17, 4096, 256, True),      # the fewest rows, the least k
    (32, 1001, 1096, True),     # a full tile of 32; N and k off the tiles
    (33, 130, 264, True),       # one row over; two columns in the second weight tile
    (64, 768, 768, True),
    (65, 769, 776, True),
    (129, 2304, 768, True),     # one row in the last token tile
    (300, 3072, 768, True),
    (512, 512, 3080, True),
    (1500, 5003, 328, True),    # several units per CTA
    (16, 4096, 256, False),
    (32, 768, 768, False),      # few rows of small weights
    (300, 768, 248, False),     # little k
])
def test_product(M, N, K, tc):
    A, Wm = _operands(M, N, K)
    out, ran = _run(A, Wm)
    assert _error(out, A, Wm) <= 1.0
    assert ran == tc
    if tc:
        # independent roundings average out, so the 2-norm sees what the bound's worst case hides: 0.7 to 2.2e-7 measured, and
        # 4.4e-6 without the three smallest of the six products of parts
        want = A.astype(np.float64) @ Wm.astype(np.float64)
        assert np.linalg.norm(out - want) <= 5e-7 * np.linalg.norm(want)


def _parts(rng, shape):
    """High, middle and low parts of values in [64, 128): each is what remains when the ones before are taken off and rounds to
    itself in bf16; sums of a stage's products of any two are exact in fp32."""
    high = rng.randint(64, 128, shape)
    return high.astype(np.float32), (rng.randint(9, 15, shape) / 64).astype(np.float32), (rng.randint(1, 64, shape) / 2 ** 17).astype(np.float32)


@pytest.mark.parametrize("M", [40, 200])  # token tiles of 64 and 128
@pytest.mark.parametrize("part", ["low of A", "low of W", "middle of both", "middle of A", "middle of W"])
def test_every_product_of_parts_counts(part, M):
    """Everything larger cancels, exactly: the result is what the named product of parts contributes."""
    rng = np.random.RandomState(M)
    N, K = 300, 1024
    A, Wm = np.zeros((M, K), np.float32), np.zeros((K, N), np.float32)
    j = np.arange(0, K, 16)  # some products a stage: its sums stay below 2^24 of their last place
    h, m, l = _parts(rng, (M, len(j)))
    h2, m2, l2 = _parts(rng, (len(j), N))
    sign = rng.choice([-1.0, 1.0], (M, len(j))).astype(np.float32)
    if part == "low of A":
        unit = rng.choice([-2.0, 1.0, 2.0], (len(j), N)).astype(np.float32)
        A[:, j], A[:, j + 1], Wm[j], Wm[j + 1] = h + m + l, -(h + m), unit, unit
        want = l.astype(np.float64) @ unit
    elif part == "low of W":
        A[:, j], A[:, j + 1], Wm[j], Wm[j + 1] = sign, -sign, h2 + m2 + l2, h2 + m2
        want = sign.astype(np.float64) @ l2
    elif part == "middle of A":
        A[:, j], A[:, j + 1], Wm[j], Wm[j + 1] = h + m, -h, h2, h2
        want = m.astype(np.float64) @ h2
    elif part == "middle of W":
        A[:, j], A[:, j + 1], Wm[j], Wm[j + 1] = sign * h, -sign * h, h2 + m2, h2
        want = (sign * h).astype(np.float64) @ m2
    else:
        A[:, j], A[:, j + 1], A[:, j + 2], A[:, j + 3] = h + m, h, h + m, h
        Wm[j], Wm[j + 1], Wm[j + 2], Wm[j + 3] = h2 + m2, -(h2 + m2), -h2, h2
        want = m.astype(np.float64) @ m2
    out, ran = _run(A, Wm)
    assert ran
    assert np.array_equal(out, want.astype(np.float32))


@pytest.mark.parametrize("scale", [-60, -100, -120, -126])
def test_small_operands(scale):
    """Values far below 2^-110, whose low parts fall under bf16's smallest subnormal (2^-133): they lose those bits, and no more."""
    A, Wm = _operands(40, 300, 520)
    A = (A.astype(np.float64) * 2.0 ** scale).astype(np.float32)
    Wm = np.ldexp(Wm, 60)
    out, ran = _run(A, Wm)
    assert ran
    want = A.astype(np.float64) @ Wm
    bound = 2.0 ** -24 * (48 + 520 / 64 + 10) * (np.abs(A).astype(np.float64) @ np.abs(Wm)) + 2.0 ** -133 * np.abs(Wm).astype(np.float64).sum(0)
    assert (np.abs(out - want) <= bound).all()


@pytest.mark.parametrize("M", [40, 200])
def test_operands_without_finite_parts(M):
    A, Wm = _operands(M, 300, 520)
    A[3, 7], A[5, 100], A[5, 101], A[20, 519] = np.inf, np.inf, -np.inf, np.nan
    Wm[300, 140] = -np.inf
    A[9, 64] = 3.4e38  # finite, but not when rounded to bf16
    A[10, 2] = -3.4e38
    Wm[64], Wm[2] = Wm[64] * 1e-3, Wm[2] * 1e-3
    out, ran = _run(A, Wm)
    assert ran
    with np.errstate(invalid="ignore"):
        want = A.astype(np.float64) @ Wm.astype(np.float64)
    finite = np.isfinite(want)
    assert np.array_equal(np.isnan(out), np.isnan(want))
    assert np.array_equal(out[~finite & ~np.isnan(want)], want[~finite & ~np.isnan(want)].astype(np.float32))
    bound = 2.0 ** -24 * 520 * (np.abs(np.where(np.isfinite(A), A, 0)).astype(np.float64) @ np.abs(np.where(np.isfinite(Wm), Wm, 0)))
    assert (np.abs(out[finite] - want[finite]) <= bound[finite]).all()


@pytest.mark.parametrize("M", [40, 200])
def test_products_out_of_range(M):
    """Finite operands whose products are not: the parts' products overflow to both infinities, the result has one."""
    A, Wm = _operands(M, 300, 520)
    A[7] = np.abs(A[7]) * 1e30 + 1e29
    Wm[:, 33] = -np.abs(Wm[:, 33]) * 1e25 - 1e24
    out, ran = _run(A, Wm)
    assert ran
    want = A.astype(np.float64) @ Wm.astype(np.float64)
    assert np.isfinite(out).sum() == out.size - 1 and out[7, 33] == -np.inf and want[7, 33] < -1e53
    bound = 2.0 ** -24 * 520 * (np.abs(A).astype(np.float64) @ np.abs(Wm))
    finite = np.isfinite(out)
    assert (np.abs(out - want)[finite] <= bound[finite]).all()


@pytest.mark.parametrize("rows,cols", [(slice(None), slice(0)), (slice(0), slice(None)), (slice(130, 131), slice(5, 6))])
def test_rows_of_nan(rows, cols):
    """All of A, all of W, a row and a column; token and weight tiles with ends past the matrices, several units per CTA."""
    A, Wm = _operands(300, 9001, 1096)
    A[rows, 1095], Wm[0, cols] = np.nan, np.nan
    out, ran = _run(A, Wm)
    assert ran
    nan = np.zeros(out.shape, bool)
    nan[rows], nan[:, cols] = True, True
    assert np.array_equal(np.isnan(out), nan)
    if not nan.all():
        a, w = np.where(np.isnan(A), 0, A), np.where(np.isnan(Wm), 0, Wm)
        assert np.abs(out - a.astype(np.float64) @ w)[~nan].max() <= 1e-4  # (of some 30)
