"""The weight GEMM where values lie far from the largest of their row: the error stays relative to sum |a||w|, output by output, as
that of fused multiply-adds in fp32 would (2^-22 of it at most over a few hundred terms, in the native format)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BAND = {"native": lambda k: 2.0 ** -22, "3xtf32": lambda k: 2.0 ** -20 + k * 2.0 ** -25, "tf32": lambda k: 2.0 ** -10, "bf16": lambda k: 2.0 ** -7}


@pytest.fixture(scope="module")
def calc(lib_path, models):
    from pet_kokkos_b200 import Calculator
    c = Calculator(*models("tiny"))
    yield c
    c.close()


def worst(calc, A, W, mode):
    ref = A.astype(np.float64) @ W.T.astype(np.float64)
    size = np.abs(A).astype(np.float64) @ np.abs(W).T.astype(np.float64)
    w = 0.0
    for transposed in (True, False):
        C = calc.gemm(A, W if transposed else np.ascontiguousarray(W.T), mode, transposed)
        assert np.isfinite(C).all()
        w = max(w, (np.abs(C - ref) / size).max())
    return w


@pytest.mark.parametrize("mode", ["native", "3xtf32", "tf32", "bf16"])
@pytest.mark.parametrize("shape", [(70, 72, 100), (300, 128, 256), (129, 512, 264), (130, 64, 1028), (300, 192, 2048), (19300, 256, 96)])
def test_rows_of_a_weight_on_scales_of_their_own(calc, shape, mode):
    """Output rows of a weight that lie up to 2^-60 below the others, and one of zeros."""
    m, n, k = shape
    rng = np.random.default_rng(m + n + k)
    A = rng.normal(size=(m, k)).astype(np.float32)
    W = rng.normal(size=(n, k)).astype(np.float32)
    W *= np.float32(2.0) ** rng.integers(-30, 31, size=(n, 1)).astype(np.float32)
    W[5] *= np.float32(1e-3)
    w = worst(calc, A, W, mode)
    assert w <= BAND[mode](k), np.log2(w)
    W[3] = 0.0
    assert (calc.gemm(A, W, mode)[:, 3] == 0.0).all()
